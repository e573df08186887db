"""Few rows per expert (the weight-streaming forward kernels): forward and backward against the CPU oracle at the edges of
their tiles -- one row, full and overfull 16-row groups, widths that end inside a 64-wide k-block, a 16-column task and a
128-row weight block -- and the inference forward bit-identical to the training one."""
import numpy as np
import pytest
import torch

from mgpt_b200 import MoELayer, synth
from oracle import oracle
from tests.util import assert_routing_exact, assert_values, dims_of, run_layer

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
    (1024, 2816, 32, 2, [[1, 2, 6, 7, 8, 20], [21, 64, 128]]),     # gate/up goes from four warps per task to one between 6 and 7
    (1024, 1032, 128, 2, [[1, 18, 36, 37, 53], [54, 300]]),        # both products do between 36 and 37; 17 k-blocks, uneven parts
    (256, 520, 16, 2, [[1, 16, 63, 64], [65, 90]]),                # four k-blocks: one part; nine: parts of 2, 2, 2 and 3
])
@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
def test_a_tokens_bits_do_not_depend_on_the_call(C, H, E, k, ranges, io):
    """The rows of a growing context keep their bits, whichever split of the reduction the number of tokens and the SM
    budget lead to, but for the one step between the kernels for few rows per expert and the others."""
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
