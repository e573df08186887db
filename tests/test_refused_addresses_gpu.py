"""Token buffers that the kernels touch 16 bytes at a time: another address is an error before those are launched, and
buffers on such boundaries work as before afterwards."""
import ctypes as ct

import pytest
import torch

from mgpt_b200 import MoELayer, _lib, synth
from mgpt_b200._lib import MoeError
from tests.test_variants_gpu import off_by_one

pytestmark = pytest.mark.gpu


def _refused(call):
    with pytest.raises(MoeError, match="byte aligned"):
        call()


@pytest.mark.parametrize("mode,io", [("fp32", torch.float32), ("bf16", torch.float32), ("bf16", torch.bfloat16)])
def test_layer_calls(mode, io):
    w = synth.Workload("addr", 37, 72, 64, 5, 2, mode)
    x, params, dy = synth.make_inputs(w, seed=4, bias_std=0.02)
    layer = MoELayer(w.C, w.H, w.E, w.k, mode=mode)
    layer.load_parameters(params)
    layer.zero_grad()
    xt, dyt = (torch.from_numpy(a).cuda().to(io) for a in (x, dy))
    off = off_by_one(torch.zeros_like(xt))
    want = layer.forward(xt).clone()
    _refused(lambda: layer.forward_into(xt, off))
    _refused(lambda: layer.forward_inference_into(xt, off))
    _refused(lambda: layer.forward_into(xt, torch.empty_like(xt), residual=off))
    y = layer.forward(xt)
    _refused(lambda: layer.backward_into(dyt, off))
    _refused(lambda: layer.backward_into(off, torch.empty_like(xt)))
    x_off = off_by_one(xt)
    layer.forward(x_off)                                        # x alone may start anywhere ...
    _refused(lambda: layer.backward(dyt))                       # ... but not for the router's weight gradient
    y = layer.forward(xt)
    assert torch.equal(y, want)
    assert torch.isfinite(layer.backward(dyt)).all()
    layer.check_status()
    layer.close()


def test_stage_calls():
    n, C, E, k = 37, 64, 4, 2
    w = synth.Workload("addr", n, C, 64, E, k, "bf16")
    x, params, _ = synth.make_inputs(w, seed=4, bias_std=0.02)
    layer = MoELayer(C, 64, E, k, mode="bf16")
    layer.load_parameters(params)
    lib, h, st = layer.lib, layer._h, layer._stream()
    xt = torch.from_numpy(x).cuda().bfloat16()
    ws = torch.empty(int(lib.mgpt_moe_stage_workspace_bytes(h, n, 1)), dtype=torch.uint8, device="cuda")
    off, nb = ct.c_size_t(), ct.c_size_t()
    _lib.check(lib.mgpt_moe_workspace_view(h, n, b"row_src", ct.byref(off), ct.byref(nb)))
    rows = torch.empty(nb.value // 4, C, dtype=torch.bfloat16, device="cuda")
    bad_rows, bad_x = off_by_one(rows), off_by_one(xt)
    args = (layer._io(xt), ws.data_ptr(), ws.numel())
    tail = (ws.data_ptr(), ws.numel(), st)
    p = lambda t: t.data_ptr()
    check = lambda rc: _lib.check(rc)
    _refused(lambda: check(lib.mgpt_moe_route(h, p(xt), n, *args, p(bad_rows), st)))
    check(lib.mgpt_moe_route(h, p(xt), n, *args, p(rows), st))
    y, dx = torch.empty_like(xt), torch.empty_like(xt)
    _refused(lambda: check(lib.mgpt_moe_combine(h, p(bad_rows), p(y), layer._io(xt), *tail)))
    _refused(lambda: check(lib.mgpt_moe_combine(h, p(rows), p(bad_x), layer._io(xt), *tail)))
    _refused(lambda: check(lib.mgpt_moe_combine_backward(h, p(rows), p(bad_x), layer._io(xt), p(rows), *tail)))
    _refused(lambda: check(lib.mgpt_moe_combine_backward(h, p(rows), p(xt), layer._io(xt), p(bad_rows), *tail)))
    _refused(lambda: check(lib.mgpt_moe_route_backward(h, p(xt), p(bad_rows), p(dx), layer._io(xt), *tail)))
    _refused(lambda: check(lib.mgpt_moe_route_backward(h, p(xt), p(rows), p(bad_x), layer._io(xt), *tail)))
    check(lib.mgpt_moe_combine(h, p(rows), p(y), layer._io(xt), *tail))
    layer.check_status()
    layer.close()


@pytest.mark.parametrize("mode,io", [("fp32", torch.float32), ("bf16", torch.bfloat16)])
def test_expert_side_rows_of_the_cuda_core_products_at_any_address(mode, io):
    """The row buffers of mgpt_moe_experts_* belong to the caller: the CUDA-core products take them wherever they start."""
    C, H, E = 72, 136, 3
    counts = torch.tensor([130, 0, 5], dtype=torch.int32, device="cuda")
    layer = MoELayer(C, H, E, 1, mode=mode, gemm_impl=1)
    gen = torch.Generator(device="cuda").manual_seed(3)
    for p in layer.get_parameters():
        p.normal_(0.0, 0.05, generator=gen)
    layer.sync_weights()
    lib, h, st, n = layer.lib, layer._h, layer._stream(), 384
    ws = torch.empty(int(lib.mgpt_moe_stage_workspace_bytes(h, n, 0)), dtype=torch.uint8, device="cuda")
    rows, d_out = torch.zeros(n, C, dtype=io, device="cuda"), torch.zeros(n, C, dtype=io, device="cuda")
    for t in (rows, d_out):
        for r0, r1 in ((0, 130), (256, 261)):
            t[r0:r1] = torch.randn(r1 - r0, C, generator=gen, device="cuda").to(io)
    runs = []
    for place in (lambda t: t.clone(), off_by_one):
        layer.zero_grad()
        x, y, dy, dx = place(rows), place(torch.zeros_like(rows)), place(d_out), place(torch.zeros_like(rows))
        _lib.check(lib.mgpt_moe_experts_forward(h, x.data_ptr(), counts.data_ptr(), 1, n, y.data_ptr(), ws.data_ptr(), ws.numel(), st))
        _lib.check(lib.mgpt_moe_experts_backward(h, dy.data_ptr(), dx.data_ptr(), ws.data_ptr(), ws.numel(), st))
        torch.cuda.synchronize()
        assert y[:130].any() and dx[256:261].any()
        runs.append([y, dx] + [p.grad.clone() for p in layer.get_parameters()])
    assert all(torch.equal(a, b) for a, b in zip(*runs))
    layer.check_status()
    layer.close()


@pytest.mark.parametrize("what,first", [("bias", 3), ("bias", 7), ("gradient", 6), ("gradient", 0)])
def test_parameters_of_the_tensor_core_products(what, first):
    """Expert biases (of gate, of down) and the gradients of Wd and Wr, which those kernels touch 16 bytes at a time."""
    n, C, H, E = 300, 64, 64, 4                                 # (too many rows for the decode kernels)
    layer = MoELayer(C, H, E, 2, mode="bf16")
    for i, p in enumerate(layer.params):
        p.normal_(0.0, 0.05)
        if what == "gradient" and (i == first or first > 0 and i >= 2 and (i - first) % 6 == 0):
            p.grad = off_by_one(torch.zeros_like(p))
        if what == "bias" and i >= 2 and (i - first) % 6 == 0:
            grad, layer.params[i] = p.grad, off_by_one(p)
            layer.params[i].grad = grad
    layer._bind()
    layer.sync_weights()
    x = torch.randn(n, C, device="cuda").bfloat16()
    if what == "bias":
        _refused(lambda: layer.forward(x))
    else:
        layer.forward(x)
        _refused(lambda: layer.backward(x))
    layer.check_status()
    layer.close()
