"""The variants that a size, an expert count or an address chooses inside the layer, each at the edges of its range: register
tiles of the exact router and its form for other shapes, top-k rounded up to a power of two, a lane's worth of experts, widths
that end inside a tile, parameter and token buffers off 16-byte boundaries, groups of warps in the block's backward."""
import ctypes as ct

import numpy as np
import pytest
import torch

from mgpt_b200 import MoELayer, _lib, synth
from oracle import oracle
from tests.util import assert_routing_exact, assert_values, dims_of, rel_l2, run_layer

pytestmark = pytest.mark.gpu


def off_by_one(t):
    """A copy of t that starts one element behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    view = buf[1:].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("n,C,E,k", [
    (1, 72, 1, 1),
    (5, 72, 3, 2),          # few (token, expert) pairs, experts not a multiple of four; plan of the router's last block
    (128, 64, 4, 2),        # the most rows that block plans
    (129, 64, 4, 2),
    (300, 136, 128, 8),     # four experts per thread, the most experts and choices
    (1300, 72, 30, 3),
    (4001, 72, 33, 4),      # two tokens per thread
    (4001, 520, 64, 2),
])
@pytest.mark.parametrize("mode,io", [("fp32", torch.float32), ("bf16", torch.float32), ("bf16", torch.bfloat16)])
def test_shapes(n, C, E, k, mode, io):
    w = synth.Workload("shapes", n, C, 64, E, k, mode)
    x, params, dy = synth.make_inputs(w, seed=n + E, bias_std=0.02)
    ref = oracle.run(dims_of(w), x, params, dy, threads=8)
    got = run_layer(w, x, params, dy, mode=mode, io=io)
    assert_routing_exact(got, ref)
    assert_values(got, ref, 1e-5 if mode == "fp32" else 2e-2, w)


@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_router_of_other_shapes_and_addresses(io):
    n, C, E, k = 333, 70, 37, 3
    rng = np.random.default_rng(1)
    x = torch.zeros(n, 72, dtype=io, device="cuda")
    Wr = torch.zeros(72, E, device="cuda")
    x[:, :C] = torch.from_numpy(rng.standard_normal((n, C)).astype(np.float32)).to(io)
    Wr[:C] = torch.from_numpy(rng.standard_normal((C, E)).astype(np.float32))
    br = torch.zeros(E, device="cuda")

    def route(x, Wr):
        out = [torch.empty(n, E, device="cuda"), torch.empty(n, E, device="cuda"),
               torch.empty(n, k, dtype=torch.int32, device="cuda"), torch.empty(n, k, device="cuda")]
        _lib.check(_lib.load().mgpt_moe_op_router(x.data_ptr(), int(io == torch.bfloat16), Wr.data_ptr(), br.data_ptr(), n, x.shape[1],
                                                  E, k, *[t.data_ptr() for t in out], torch.cuda.current_stream().cuda_stream))
        return out

    want = route(x, Wr)                       # two channels of zeros add nothing, exactly
    for got in (route(x[:, :C].contiguous(), Wr[:C]), route(off_by_one(x), off_by_one(Wr))):
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("n", [9, 333])
def test_tokens_off_16_byte_boundaries(n):
    """FP32 tokens of a BF16 layer, forward only: the decode kernels' size and the tensor-core products'."""
    w = synth.Workload("off", n, 136, 200, 5, 2, "bf16")
    x, params, _ = synth.make_inputs(w, seed=9, bias_std=0.02)
    layer = MoELayer(w.C, w.H, w.E, w.k, mode="bf16")
    layer.load_parameters(params)
    xt = torch.from_numpy(x).cuda()
    want = layer.forward_inference(xt)
    assert torch.equal(layer.forward_inference(off_by_one(xt)), want)
    assert torch.equal(layer.forward(off_by_one(xt)), want)
    layer.check_status()


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
def test_parameters_off_16_byte_boundaries(mode):
    w = synth.Workload("off", 333, 136, 200, 5, 2, mode)
    x, params, dy = synth.make_inputs(w, seed=9, bias_std=0.02)
    xt, dyt = torch.from_numpy(x).cuda(), torch.from_numpy(dy).cuda()
    out = []
    for place in (lambda t: t, off_by_one):
        layer = MoELayer(w.C, w.H, w.E, w.k, mode=mode)
        layer.params = [place(p) for p in layer.params]
        for p in layer.params:
            p.grad = place(torch.zeros_like(p))
        layer._bind()
        layer.load_parameters(params)
        if mode == "fp32":                    # (the BF16 products want the biases on 16-byte boundaries)
            out.append([layer.forward(xt), layer.backward(dyt)])
        for i, p in enumerate(layer.params):
            if mode == "fp32" and place is off_by_one:
                assert rel_l2(p.grad.cpu().numpy(), grads[i].cpu().numpy()) <= 1e-6
            p.grad.copy_(torch.sin(torch.arange(p.numel(), device="cuda", dtype=torch.float32)).view(p.shape) if mode == "bf16"
                         else p.grad if place is not off_by_one else grads[i])
        grads = [p.grad for p in layer.params]
        layer.opt_m = [place(torch.zeros_like(p)) for p in layer.params]
        layer.opt_v = [place(torch.zeros_like(p)) for p in layer.params]
        m, v = ((ct.c_void_p * len(layer.params))(*[t.data_ptr() for t in ts]) for ts in (layer.opt_m, layer.opt_v))
        _lib.check(layer.lib.mgpt_moe_bind_optimizer_state(layer._h, m, v, len(layer.params)))
        layer.adamw_step(1)
        layer.check_status()
        out.append(list(layer.params) + layer.opt_m + layer.opt_v)
    half = len(out) // 2
    for a, b in zip(out[:half], out[half:]):
        assert all(torch.equal(s, t) for s, t in zip(a, b))


@pytest.mark.parametrize("C,n", [(8, 3), (264, 700), (1536, 9), (1544, 9), (3080, 9), (6152, 9), (12288, 5)])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_block_backward_widths(C, n, io):
    w = synth.Workload("blk", n, C, 8, 2, 1, "bf16" if io == torch.bfloat16 else "fp32")
    x1, params, dout = synth.make_inputs(w, seed=C, bias_std=0.02)
    if io == torch.bfloat16:
        x1, dout = synth.bf16_round(x1), synth.bf16_round(dout)
    gamma = (1.0 + 0.1 * np.random.default_rng(2).standard_normal(C)).astype(np.float32)
    layer = MoELayer(C, w.H, w.E, w.k, mode=w.dtype, lb_alpha=w.alpha)
    layer.load_parameters(params)
    tol = 2e-5 if io == torch.float32 else 2e-2
    got = []
    for place in (lambda t: t, off_by_one):
        layer.zero_grad()
        g = place(torch.from_numpy(gamma).cuda())                # (its address chooses between 16-byte and single accesses)
        x, d = torch.from_numpy(x1).cuda().to(io), torch.from_numpy(dout).cuda().to(io)
        dg = torch.zeros(C, device="cuda")
        layer.block_forward(x, g)
        ln2 = layer.block_input().float().cpu().numpy()
        d_x1 = layer.block_backward(g, d, dg)
        moe = oracle.run(dims_of(w), ln2, params, dout, threads=8)
        _, _, dn, dgam = oracle.rmsnorm(x1, gamma, moe["dx"])
        assert rel_l2(d_x1.float().cpu().numpy(), dout + dn) <= tol
        assert rel_l2(dg.cpu().numpy(), dgam) <= tol
        got.append(d_x1)
    layer.check_status()
    assert all(rel_l2(b.float().cpu().numpy(), got[0].float().cpu().numpy()) <= 1e-6 for b in got)
    layer.close()
