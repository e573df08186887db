"""Weight gradients on CTA pairs, which 512 rows per expert or more take: against the products of the very operands the kernel
read (the layer's own buffers), so that only the order of FP32 sums separates the two."""
import pytest
import torch

from mgpt_b200 import MoELayer

pytestmark = pytest.mark.gpu

# FP32 sums of up to 3000 products in two orders: n * 2^-24 * sum|ab| bounds each, and sum|ab| / |sum ab| is about sqrt(n) here, so
# 3000^1.5 * 6e-8 = 1e-2 at the very worst and ~sqrt(n) * 6e-8 = 3e-6 as rounding goes.  A 64-row block too many or too few
# changes a sum by a few percent.
TOL = 1e-4


@pytest.mark.parametrize("n,C,H,E,k,skew", [
    (1300, 512, 512, 4, 2, False),      # whole tiles
    (1100, 640, 712, 4, 2, False),      # an odd number of 128-channel tiles; H ends inside a tile, inside a 64-column box
    (1100, 328, 1376, 4, 2, False),     # C not a multiple of 64; last column tiles of 72 and of 96
    (700, 1024, 264, 1, 1, False),      # the narrowest H that pairs take, one expert
    (2100, 320, 384, 8, 2, True),       # experts without rows, one with a quarter of all
    (8192, 264, 272, 128, 8, False),    # the most experts
])
@pytest.mark.parametrize("store", [False, True])
@pytest.mark.parametrize("sms", [0, 5])
def test_against_the_operands(n, C, H, E, k, skew, store, sms):
    gen = torch.Generator(device="cuda").manual_seed(n + C)
    layer = MoELayer(C, H, E, k, mode="bf16")
    for p in layer.get_parameters():
        p.normal_(0.0, 0.02, generator=gen)
        p.grad.normal_(0.0, 1.0, generator=gen)
    if skew:
        layer.get_parameters()[1].copy_(torch.tensor([[9.0] + [0.0] * (E - 4) + [-99.0] * 3], device="cuda"))
    layer.sync_weights()
    before = [p.grad.clone() for p in layer.get_parameters()]
    layer.set_weight_grad_overwrite(store)
    layer.lib.mgpt_moe_set_sm_budget(layer._h, sms)
    x, dy = (torch.randn(n, C, generator=gen, device="cuda").bfloat16() for _ in range(2))
    layer.forward(x)
    layer.backward(dy)
    layer.check_status()
    off = layer.workspace_view("padded_offsets", torch.int32).tolist()
    counts = layer.get_expert_counts()
    assert n * k >= 512 * E and (not skew or 0 in counts)
    Xg, dYg = (layer.workspace_view(b, torch.bfloat16).view(-1, C).float() for b in ("Xg", "dYg"))
    Hh, dG, dU = (layer.workspace_view(b, torch.bfloat16).view(-1, H).float() for b in ("Hh", "dG", "dU"))
    for e in range(E):
        r = slice(off[e], off[e + 1])
        want = [Xg[r].double().T @ dG[r].double(), dG[r].double().sum(0), Xg[r].double().T @ dU[r].double(), dU[r].double().sum(0),
                Hh[r].double().T @ dYg[r].double(), dYg[r].double().sum(0)]
        for i, v in enumerate(want):
            p, g0 = layer.get_parameters()[2 + 6 * e + i], before[2 + 6 * e + i]
            stored = store and i % 2 == 0               # (bias gradients are always added)
            got = p.grad.double() - (0 if stored else g0.double())
            # what an addition to g0 rounds away: half a ulp of values of ~1 each
            slack = 0.0 if stored else 2.0 ** -23 * p.grad.numel() ** 0.5
            assert (got - v.view(p.shape)).norm() <= TOL * v.norm() + slack, (e, i)
    layer.close()
