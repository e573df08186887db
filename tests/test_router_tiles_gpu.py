"""The exact router's register tiles (experts x tokens per thread), which the number of tokens and the padded number of experts
choose: each of them, with rows that end inside a stage and experts that end inside a lane's share."""
import pytest
import torch

from mgpt_b200 import _lib, synth
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


@pytest.mark.parametrize("share,E,k", [
    (40, 4, 2), (300, 3, 1),                        # tokens per SM: 1x4, one row of tokens per warp and two
    (33, 7, 2), (150, 8, 8),                        # 2x4, one and two
    (20, 12, 3), (100, 9, 2), (140, 11, 2),         # 4x3, one, two and three
    (40, 16, 2), (90, 13, 2), (150, 16, 4),         # 8x2, two and three; 4x4, three
    (30, 24, 2), (120, 21, 2), (70, 20, 2),         # 8x3, one and four; 4x5, two
    (40, 32, 8), (60, 29, 2),                       # 16x2, three; 8x4, two
    (8, 48, 2), (30, 43, 3), (45, 40, 2),           # 16x3, one and two; 8x5, two
    (20, 64, 2), (45, 57, 2),                       # 32x2, three; 16x4, three
    (7, 96, 2), (30, 81, 2), (30, 80, 8), (47, 66, 2),      # 32x3, one and four; 16x5, two and three
    (30, 128, 2), (12, 101, 8),                     # 32x4, four and two
])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_rows_of_a_warp(share, E, k, io):
    """Several rows of tokens per warp, the last one with tokens for some of the warps only."""
    w = synth.Workload("rows", 148 * share - 3, 136, 8, E, k, "bf16")
    x, params, _ = synth.make_inputs(w, seed=share + E, bias_std=0.02)
    if io == torch.bfloat16:
        x = synth.bf16_round(x)
    ref = oracle.run(dims_of(w), x, params, None, threads=8)
    got = run_layer(w, x, params, None, mode="bf16", io=io)
    assert not got["screened"]
    assert_routing_exact(got, ref)
    got["layer"].close()


def test_experts_between_powers_of_two_cost_their_share():
    """Device times against the next power of two's.  Padded up to it they took 1.0 to 1.1 times as long, and 2.2 to 2.4 times
    where a row of Wr is no multiple of 16 bytes; now 0.77, 0.84, 0.77 and 1.2, 1.1."""
    lib = _lib.load()
    stream = torch.cuda.Stream()

    def us(n, E, C=512, k=2):
        x, Wr, br = torch.randn(n, C, device="cuda"), torch.randn(C, E, device="cuda") * 0.02, torch.zeros(E, device="cuda")
        probs, idx, top = torch.empty(n, E, device="cuda"), torch.empty(n, k, dtype=torch.int32, device="cuda"), torch.empty(n, k, device="cuda")
        torch.cuda.synchronize()
        best = float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(400000)               # the calls are all enqueued before the first one starts
            a.record()
            for _ in range(20):
                _lib.check(lib.mgpt_moe_op_router(x.data_ptr(), 0, Wr.data_ptr(), br.data_ptr(), n, C, E, k, None, probs.data_ptr(),
                                                  idx.data_ptr(), top.data_ptr(), stream.cuda_stream))
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 50)
        return best

    with torch.cuda.stream(stream):
        for n, E, next_E, most in ((32768, 8, 16, 0.9), (300, 31, 32, 1.7), (32768, 48, 64, 0.95), (32768, 80, 128, 0.95),
                                   (32768, 127, 128, 1.5)):
            t, u = us(n, E), us(n, next_E)
            assert t < most * u, (n, E, t, u)
