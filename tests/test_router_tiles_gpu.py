"""The exact router's register tiles (experts x tokens per thread), which the number of tokens and the padded number of experts
choose: each of them, with rows that end inside a stage and experts that end inside a lane's share."""
import pytest
import torch

from mgpt_b200 import synth
from oracle import oracle
from tests.util import assert_routing_exact, dims_of, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,C,E,k", [
    (2368, 72, 5, 2), (2369, 264, 16, 3), (4737, 520, 7, 1), (9473, 72, 16, 2),         # 16 experts: 1x1, 2x1, 2x2, 4x2
    (1184, 520, 32, 2), (1185, 264, 17, 8), (2369, 72, 32, 2), (4737, 72, 31, 2),       # 32: the same
    (592, 1032, 64, 2), (1185, 264, 33, 4), (2369, 72, 64, 8),                          # 64: 2x1, 2x2, 4x2
    (1184, 264, 65, 2), (1185, 72, 127, 3),                                             # 128: 4x1, 4x2
])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_every_tile(n, C, E, k, io):
    w = synth.Workload("tiles", n, C, 8, E, k, "bf16")
    x, params, _ = synth.make_inputs(w, seed=n + E, bias_std=0.02)
    if io == torch.bfloat16:
        x = synth.bf16_round(x)
    ref = oracle.run(dims_of(w), x, params, None, threads=8)
    got = run_layer(w, x, params, None, mode="bf16", io=io)
    assert_routing_exact(got, ref)
    got["layer"].close()
