"""Routing-side workspaces (mgpt_moe_route) under the views and the saved routing of the whole layer: one layout for every
kind of workspace, also at the sizes where the plan lists row groups."""
import ctypes as ct

import pytest
import torch

from mgpt_b200 import MoELayer, _lib, synth
from tests.util import assert_plan_equal, plan_reference

pytestmark = pytest.mark.gpu

VIEWS = ("counts", "offsets", "padded_offsets", "tile_expert", "n_tiles", "map", "pos", "row_src", "status")


def _routed(n, E, k=2, C=256, H=256):
    """A whole layer whose last call was mgpt_moe_route over n tokens, its tokens and the workspace."""
    w = synth.Workload("views", n, C, H, E, k, "bf16")
    x, params, _ = synth.make_inputs(w, seed=n, bias_std=0.02)
    layer = MoELayer(C, H, E, k, mode="bf16")
    layer.load_parameters(params)
    xt = torch.from_numpy(x).cuda().bfloat16()
    lib, h = layer.lib, layer._h
    # room for the whole layer's buffers, so that a view outside the routing side's part still lies in the tensor
    ws = torch.zeros(int(lib.mgpt_moe_workspace_bytes(h, n)), dtype=torch.uint8, device="cuda")
    off, nb = ct.c_size_t(), ct.c_size_t()

    def view(name):
        _lib.check(lib.mgpt_moe_workspace_view(h, n, name.encode(), ct.byref(off), ct.byref(nb)))
        return ws[off.value: off.value + nb.value].view(torch.int32)

    send = torch.empty(view("row_src").numel(), C, dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.mgpt_moe_route(h, xt.data_ptr(), n, layer._io(xt), ws.data_ptr(), ws.numel(), send.data_ptr(), layer._stream()))
    torch.cuda.synchronize()
    layer._n = n
    return layer, xt, ws, send, view


@pytest.mark.parametrize("n,E", [(1, 8), (8, 32), (128, 32), (129, 32), (300, 64)])
def test_views_of_a_routing_side_workspace(n, E):
    layer, xt, ws, send, view = _routed(n, E)
    top_idx = view("top_idx").cpu().numpy()
    ref = plan_reference(top_idx, E)
    assert_plan_equal({k: view(k) for k in VIEWS}, ref, n * 2)
    pos = view("pos").long()
    assert torch.equal(send[pos].view(n, 2, -1), xt[:, None].expand(-1, 2, -1))      # the rows lie where the view says
    layer.check_status()
    layer.close()


@pytest.mark.parametrize("E,k", [(8, 2), (128, 1), (128, 8)])
def test_sizes_never_shrink_as_the_tokens_grow(E, k):
    """A workspace for the largest call serves every smaller one."""
    layer = MoELayer(64, 64, E, k, mode="bf16")
    lib, h = layer.lib, layer._h
    sizes = {"layer": lambda n: lib.mgpt_moe_workspace_bytes(h, n), "inference": lambda n: lib.mgpt_moe_inference_workspace_bytes(h, n),
             "routing side": lambda n: lib.mgpt_moe_stage_workspace_bytes(h, n, 1),
             "expert side": lambda n: lib.mgpt_moe_stage_workspace_bytes(h, n, 0), "routing": lambda n: lib.mgpt_moe_routing_bytes(h, n)}
    for what, size in sizes.items():
        s = [int(size(n)) for n in range(8 * E // k + 40)]
        assert all(a <= b for a, b in zip(s, s[1:])), what
    layer.close()


@pytest.mark.parametrize("n,E", [(8, 32), (300, 64)])
def test_saved_routing_of_a_routing_side_call(n, E):
    """Routing saved after mgpt_moe_route feeds the whole layer's recompute: the outputs of its own forward."""
    layer, xt, ws, send, view = _routed(n, E)
    saved = layer.save_routing()
    y = torch.empty_like(xt)
    layer.recompute_into(xt, y, saved)
    assert torch.equal(y, layer.forward(xt))
    layer.check_status()
    layer.close()
