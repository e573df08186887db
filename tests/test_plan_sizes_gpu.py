"""Dispatch plans of many row blocks (mgpt_moe_op_plan): the same plan on both sides of the size from which the block
histograms are scanned by a kernel of their own, and a cost that grows with the rows, not with their square."""
import ctypes as ct

import pytest
import torch

from mgpt_b200 import _lib
from tests.util import PLAN_OUTPUTS, plan_buffers, plan_row_cap

pytestmark = pytest.mark.gpu


def _plan(top_idx, E):
    lib, n = _lib.load(), top_idx.numel()
    bufs = plan_buffers(n, E)
    size = int(lib.mgpt_moe_op_plan_scratch_bytes(n, E))
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")

    def call():
        _lib.check(lib.mgpt_moe_op_plan(top_idx.data_ptr(), n, E, *[bufs[k].data_ptr() for k in PLAN_OUTPUTS[:-1]],
                                        plan_row_cap(n, E), bufs["status"].data_ptr(), scratch.data_ptr(), size,
                                        ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return bufs, call


@pytest.mark.parametrize("n_rows", [255 * 1024, 255 * 1024 + 1, 300_001, (1 << 21) + 77])
@pytest.mark.parametrize("E", [1, 33, 128])
def test_plan_of_many_blocks(n_rows, E):
    gen = torch.Generator(device="cuda").manual_seed(n_rows + E)
    top_idx = (torch.rand(n_rows, generator=gen, device="cuda") ** 2 * E).int().clamp_(0, E - 1)      # skewed
    if E > 2:
        top_idx[top_idx == 1] = 0                                                                     # an empty expert
    bufs, call = _plan(top_idx, E)
    call()
    counts = torch.bincount(top_idx, minlength=E).int()
    offsets = counts.cumsum(0).int() - counts
    padded = (counts + 127) // 128 * 128
    poff = torch.cat([padded.new_zeros(1), padded.cumsum(0).int()])
    order = torch.sort(top_idx, stable=True).indices
    expert = top_idx[order].long()
    row = (poff[expert] + torch.arange(n_rows, device="cuda") - offsets[expert]).int()
    nt = int(poff[-1]) // 128
    row_src = torch.full((nt * 128,), -1, dtype=torch.int32, device="cuda")
    row_src[row.long()] = order.int()
    pos = torch.empty_like(top_idx)
    pos[order] = row
    want = {"counts": counts, "offsets": offsets, "padded_offsets": poff, "n_tiles": poff.new_tensor([nt]), "map": order.int(),
            "pos": pos, "row_src": row_src, "status": poff.new_zeros(1),
            "tile_expert": torch.repeat_interleave(torch.arange(E, device="cuda", dtype=torch.int32), padded // 128)}
    for key, w in want.items():
        assert torch.equal(bufs[key][:w.numel()], w), key


def test_plan_cost_grows_with_the_rows():
    """Eight times the rows may take at most twice eight times the time (with every block summing all blocks' histograms it
    was some fifty times)."""
    ms = {}
    for n in (1 << 21, 1 << 24):
        top_idx = (torch.arange(n, device="cuda", dtype=torch.int32) * 7919) % 64
        bufs, call = _plan(top_idx, 64)
        for _ in range(3):
            call()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            call()
        b.record()
        b.synchronize()
        ms[n] = a.elapsed_time(b) / 5
    assert ms[1 << 24] <= 16 * ms[1 << 21], ms
