"""Few rows per expert (the weight-streaming forward kernels): forward and backward against the CPU oracle at the edges of
their tiles -- one row, full and overfull 16-row groups, widths that end inside a 64-wide k-block, a 16-column task and a
128-row weight block -- and the inference forward bit-identical to the training one."""
import numpy as np
import pytest
import torch

from mgpt_b200 import synth
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
