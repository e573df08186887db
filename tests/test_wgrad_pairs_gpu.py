"""Weight gradients on CTA pairs, which 512 rows per expert or more take: against the products of the very operands the kernel
read (the layer's own buffers), so that only the order of FP32 sums separates the two."""
import pytest
import torch

from mgpt_b200 import MoELayer, _lib

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


@pytest.mark.parametrize("C,H", [(512, 384), (328, 712)])       # the maps of Xg and dYg by column blocks, and not
@pytest.mark.parametrize("counts", [
    [[700, 0, 129, 0], [1, 0, 900, 640], [300, 0, 0, 320]],     # three sources; segments without rows, an expert without any
    [[130, 1000, 64, 640], [0, 128, 1, 300]],
])
@pytest.mark.parametrize("store", [False, True])
def test_rows_in_segments(C, H, counts, store):
    """The expert side of an expert-parallel layer: an expert's rows lie in one segment per source.  Against the single-CTA
    kernel (which one SM takes) on the same rows, and against FP64 products of operands rounded as the layer rounds them."""
    E, n_src = len(counts[0]), len(counts)
    pad = [[(c + 127) // 128 * 128 for c in row] for row in counts]
    n_rows = sum(map(sum, pad))
    assert n_rows >= 512 * E
    gen = torch.Generator(device="cuda").manual_seed(C)
    rows, d_out = torch.zeros(2, n_rows, C, device="cuda", dtype=torch.bfloat16)
    where = [[] for _ in range(E)]
    at = 0
    for s in range(n_src):
        for e in range(E):
            for t in (rows, d_out):
                t[at: at + counts[s][e]] = torch.randn(counts[s][e], C, generator=gen, device="cuda").bfloat16()
            where[e] += range(at, at + counts[s][e])
            at += pad[s][e]
    seg = torch.tensor(counts, dtype=torch.int32, device="cuda")
    weights = None
    got = []
    for sms in (0, 7, 1):
        layer = MoELayer(C, H, E, 1, mode="bf16")
        gen.manual_seed(H)
        for p in layer.get_parameters():
            p.normal_(0.0, 0.02, generator=gen)
            p.grad.normal_(0.0, 1.0, generator=gen)
        layer.sync_weights()
        before = [p.grad.clone() for p in layer.get_parameters()]
        weights = [p.clone() for p in layer.get_parameters()]
        layer.set_weight_grad_overwrite(store)
        lib, h, st = layer.lib, layer._h, layer._stream()
        lib.mgpt_moe_set_sm_budget(h, sms)
        size = lib.mgpt_moe_stage_workspace_bytes(h, n_rows, 0)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        out, d_in = torch.empty_like(rows), torch.empty_like(rows)
        _lib.check(lib.mgpt_moe_experts_forward(h, rows.data_ptr(), seg.data_ptr(), n_src, n_rows, out.data_ptr(), ws.data_ptr(), size, st))
        _lib.check(lib.mgpt_moe_experts_backward(h, d_out.data_ptr(), d_in.data_ptr(), ws.data_ptr(), size, st))
        layer.check_status()
        got.append([p.grad.double() - (0 if store and i >= 2 and i % 2 == 0 else g.double())
                    for i, (p, g) in enumerate(zip(layer.get_parameters(), before))])
        layer.close()
    for e in range(E):
        x, dy = rows[where[e]].double(), d_out[where[e]].double()
        wg, bg, wu, bu, wd, _ = (w.double() for w in weights[2 + 6 * e: 8 + 6 * e])
        wg, wu, wd = (w.bfloat16().double() for w in (wg, wu, wd))
        g, u = x @ wg + bg, x @ wu + bu
        sig = torch.sigmoid(g)
        dh = dy @ wd.T
        hh, dg, du = ((t.bfloat16().double()) for t in (g * sig * u, dh * u * sig * (1 + g * (1 - sig)), dh * g * sig))
        want = [x.T @ dg, dg.sum(0), x.T @ du, du.sum(0), hh.T @ dy, dy.sum(0)]
        for i, v in enumerate(want):
            one = got[2][2 + 6 * e + i]
            slack = 0.0 if store and i % 2 == 0 else 2.0 ** -23 * one.numel() ** 0.5
            for pairs in got[:2]:
                a = pairs[2 + 6 * e + i]
                assert (a - one).norm() <= TOL * one.norm() + slack, (e, i)
                # (BF16 factors of dG and dU, rounded once more than here: 2^-9 of each product)
                assert (a - v.view(a.shape)).norm() <= 1e-2 * v.norm() + slack, (e, i)
