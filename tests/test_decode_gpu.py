"""Few rows per expert (the weight-streaming forward kernels): forward and backward against the CPU oracle at the edges of
their tiles -- one row, full and overfull 16-row groups, widths that end inside a 64-wide k-block, a 16-column task and a
128-row weight block -- and the inference forward bit-identical to the training one."""
import numpy as np
import pytest
import torch

from mgpt_b200 import MoELayer, synth
from oracle import oracle
from tests.util import assert_routing_exact, assert_values, dims_of, rel_l2, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,C,H,E,k,crowd", [
    (1, 64, 64, 4, 2, False),
    (7, 72, 200, 8, 3, False),
    (32, 1032, 136, 16, 4, False),        # 8 rows per expert, the most these kernels take on average
    (33, 520, 520, 17, 1, True),          # one expert with every row: three groups, the last of one row
    (16, 256, 1400, 128, 8, False),
])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_few_rows_per_expert(n, C, H, E, k, crowd, io):
    w = synth.Workload("few", n, C, H, E, k, "bf16")
    x, params, dy = synth.make_inputs(w, seed=3 + n, bias_std=0.02)
    if crowd:
        params[1][0, 5] = np.float32(64.0)
    ref = oracle.run(dims_of(w), x, params, dy, threads=4)
    got = run_layer(w, x, params, dy, mode="bf16", io=io)
    assert_routing_exact(got, ref)
    assert_values(got, ref, 2e-2, w)
    layer = got["layer"]
    xt = torch.from_numpy(x).cuda().to(io)
    assert torch.equal(layer.forward_inference(xt), layer.forward(xt))
    layer.check_status()


@pytest.mark.parametrize("C,H,E,k,ranges", [
    # (a range: token counts that take the same kernels)
    (1024, 2816, 32, 2, [[1, 2, 6, 7, 8, 33], [34, 64, 128]]),     # from 7 tokens on every warp could have two tasks of its own
    (1024, 1032, 128, 2, [[1, 18, 36, 37, 70], [71, 300]]),        # from 37; 17 k-blocks in uneven parts
    (256, 520, 16, 2, [[1, 16, 63, 64], [65, 90]]),                # four k-blocks: one warp; nine: parts of 2, 2, 2 and 3
])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_a_tokens_bits_do_not_depend_on_the_call(C, H, E, k, ranges, io):
    """The rows of a growing context keep their bits, whatever the number of tokens and the SM budget, but for the one step
    between the kernels for few rows per expert and the others."""
    n_all = ranges[-1][-1]
    w = synth.Workload("grow", n_all, C, H, E, k, "bf16")
    x, params, _ = synth.make_inputs(w, seed=29, bias_std=0.02)
    layer = MoELayer(C, H, E, k, mode="bf16")
    layer.load_parameters(params)
    xt = torch.from_numpy(x).cuda().to(io)
    for steps in ranges:
        full = layer.forward_inference(xt[:steps[-1]].contiguous()).clone()
        for n in steps:
            assert torch.equal(layer.forward_inference(xt[:n].contiguous()), full[:n]), n
    few = layer.forward_inference(xt[:8].contiguous()).clone()
    for sms in (1, 40):
        layer.lib.mgpt_moe_set_sm_budget(layer._h, sms)
        assert torch.equal(layer.forward_inference(xt[:8].contiguous()), few), sms
    layer.check_status()
    layer.close()


@pytest.mark.parametrize("n,C,H,E,k", [(1, 64, 64, 4, 2), (40, 264, 200, 16, 2), (130, 72, 1032, 17, 1)])
def test_padding_rows_of_a_workspace_full_of_nans(n, C, H, E, k):
    """Backward multiplies the padding rows of what forward keeps by zeros: they have to be finite whatever was there."""
    w = synth.Workload("pads", n, C, H, E, k, "bf16")
    x, params, dy = synth.make_inputs(w, seed=n, bias_std=0.02)
    layer = MoELayer(C, H, E, k, mode="bf16")
    layer.load_parameters(params)
    xt, dyt = torch.from_numpy(x).cuda().bfloat16(), torch.from_numpy(dy).cuda().bfloat16()
    runs = []
    for fill in (0, 255):
        layer.zero_grad()
        layer._workspace(n).fill_(fill)
        y = layer.forward(xt).clone()
        runs.append([y, layer.backward(dyt).clone()] + [p.grad.clone() for p in layer.get_parameters()])
    rows = int(layer.workspace_view("n_tiles", torch.int32)[0]) * 128
    pads = layer.workspace_view("row_src", torch.int32)[:rows] < 0
    for name in ("Xg", "Hh"):
        assert not layer.workspace_view(name, torch.bfloat16).view(-1, C if name == "Xg" else H)[:rows][pads].any(), name
    for name in ("G", "U"):
        t = layer.workspace_view(name, torch.bfloat16)[:rows * H].view(-1, H // 8, 128, 8).permute(0, 2, 1, 3).reshape(-1, H)
        assert not t[pads].any(), name
    for a, b in zip(*runs):
        assert torch.isfinite(b).all()
        torch.testing.assert_close(b.float(), a.float(), rtol=1e-5, atol=1e-6)      # (only the order of FP32 atomics differs)
    layer.check_status()
    layer.close()


@pytest.mark.parametrize("n,C,H,E,k,crowd", [
    (1, 64, 64, 4, 2, False),
    (7, 72, 200, 8, 3, False),
    (32, 1032, 136, 16, 4, False),
    (33, 520, 520, 17, 1, True),
    (6, 1024, 2816, 32, 2, False),
    (33, 1024, 2816, 32, 2, False),       # the most tokens of this shape
])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_buffers_against_the_cuda_core_products(n, C, H, E, k, crowd, io):
    """What these kernels write, buffer by buffer, against the CUDA-core products on the same BF16 data, at the bar of the
    tensor-core ones: each side's stored value is within 2^-9 of its FP32 sum, and the cross-check makes Hh and the factors
    from gate and up as it has stored them, so three such roundings lie between the two at most."""
    w = synth.Workload("cross", n, C, H, E, k, "bf16")
    x, params, _ = synth.make_inputs(w, seed=5 + n, bias_std=0.02)
    if crowd:
        params[1][0, 5] = np.float32(64.0)
    xt = torch.from_numpy(x).cuda().to(io)
    got = {}
    for impl in (0, 1):
        layer = MoELayer(C, H, E, k, mode="bf16", gemm_impl=impl)
        layer.load_parameters(params)
        y = layer.forward(xt)
        real = layer.workspace_view("row_src", torch.int32) >= 0
        real[int(layer.workspace_view("n_tiles", torch.int32)[0]) * 128:] = False
        bufs = {"y": y.float()}
        for name, width in (("G", H), ("U", H), ("Hh", H), ("Yg", C)):
            t = layer.workspace_view(name, torch.bfloat16)
            if impl == 0 and name in "GU":          # [row tile][8-column chunk][128 rows][8]
                t = t.view(-1, width // 8, 128, 8).permute(0, 2, 1, 3).reshape(-1, width)
            bufs[name] = t.view(-1, width)[real].double()
        if impl == 1:
            g, u = bufs["G"], bufs["U"]
            sig = torch.sigmoid(g)
            bufs["G"], bufs["U"] = u * sig * (1.0 + g * (1.0 - sig)), g * sig
        got[impl] = bufs
        layer.check_status()
        layer.close()
    for name, want in got[1].items():
        err = rel_l2(got[0][name].cpu().numpy(), want.cpu().numpy())
        assert err < 6e-3, (name, err)
