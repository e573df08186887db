"""The SwiGLU factors that forward keeps for backward, where the up product is infinite: dG = dHh * u*sig*(1 + g*(1 - sig)) stays
infinite with the sign of its factors, as in the reference's order of operations (utils/Tensor.cpp:2020-2027)."""
import numpy as np
import pytest
import torch

from mgpt_b200 import MoELayer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate", [-1.0, -0.25, 0.0, 0.25, 1.0, 40.0])
@pytest.mark.parametrize("up", [np.inf, -np.inf])
def test_infinite_up_product(gate, up):
    C = H = 64
    n, unit = 128, 5                               # one whole tile: padding rows would meet the infinite bias too
    layer = MoELayer(C, H, 1, 1, mode="bf16")
    Wg, bg, Wu, bu, Wd, bd = layer.get_parameters()[2:]
    Wd.fill_(0.25)
    bg[0, unit] = gate
    bu[0, unit] = float(up)
    layer.sync_weights()
    x = torch.randn(n, C, device="cuda").bfloat16()
    layer.forward(x)
    layer.backward(torch.ones_like(x))             # dHh = 0.25 * C for every unit
    layer.check_status()
    got = layer.get_parameters()[3].grad.flatten()[unit].item()
    sig = 1.0 / (1.0 + np.exp(-gate))
    assert got == up * np.sign(1.0 + gate * (1.0 - sig)), got
    layer.close()
