"""FP32 products whose k loop several CTAs of a cluster share: two, four and eight of them, ends of rows, columns and k inside a
tile, parameters off 16-byte boundaries."""
import pytest
import torch

from mgpt_b200 import MoELayer, synth
from oracle import oracle
from tests.util import assert_routing_exact, assert_values, dims_of, rel_l2, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,C,H,E,k", [
    (30, 64, 1032, 2, 2),       # one tile of columns: eight CTAs
    (64, 264, 1024, 8, 2),      # four; C ends inside a tile
    (500, 128, 520, 8, 2),      # two in dXg; the shortest k that is shared
    # gate/up (both sums through the same shared memory) and dHh share theirs from C = 256 on: eight, four and two CTAs, H ends
    # inside a second and a third tile of columns
    (30, 1032, 72, 2, 2), (64, 520, 136, 4, 2), (64, 264, 136, 4, 2),
])
def test_shared_k_loops(n, C, H, E, k):
    w = synth.Workload("clusters", n, C, H, E, k, "fp32")
    x, params, dy = synth.make_inputs(w, seed=n + C, bias_std=0.02)
    ref = oracle.run(dims_of(w), x, params, dy, threads=8)
    got = run_layer(w, x, params, dy, mode="fp32")
    assert_routing_exact(got, ref)
    assert_values(got, ref, 1e-5, w)

    # the same from parameters that allow single accesses only: the same sums in the same order
    layer = MoELayer(C, H, E, k, mode="fp32", lb_alpha=w.alpha)
    layer.params = [torch.empty(p.numel() + 1, device="cuda")[1:].view(p.shape) for p in layer.params]
    for p in layer.params:
        p.grad = torch.zeros(p.numel() + 1, device="cuda")[1:].view(p.shape)
    layer._bind()
    layer.load_parameters(params)
    y = layer.forward(torch.from_numpy(x).cuda())
    dx = layer.backward(torch.from_numpy(dy).cuda())
    layer.check_status()
    assert rel_l2(y.cpu().numpy(), got["y"]) <= 1e-6 and rel_l2(dx.cpu().numpy(), got["dx"]) <= 1e-6
    layer.close()
    got["layer"].close()


def test_more_tiles_than_expected():
    """Clusters that may not fit on the SMs in one round are not made: 412 tokens, 18 row tiles expected and 24 in this routing,
    took 1.3 times as long as 448 tokens with as many tiles, one CTA each."""
    C = H = 256
    E = 12

    def us(n):
        layer = MoELayer(C, H, E, 2, mode="fp32")
        for p in layer.get_parameters():
            p.normal_(0.0, 0.02)
        router = layer.get_parameters()[0]
        router.zero_()
        router[:E] = torch.eye(E, device="cuda")
        layer.sync_weights()
        t = torch.arange(n, device="cuda")
        x = torch.randn(n, C, device="cuda")
        x[:, :E] = 0.0
        x[t, t % E] = 8.0                           # every expert gets as many rows
        x[t, (t + 1) % E] = 6.0
        y, dx = torch.empty_like(x), torch.empty_like(x)
        best = float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(2000000)              # the calls are all enqueued before the first one starts
            a.record()
            for _ in range(20):
                layer.forward_into(x, y)
                layer.backward_into(x, dx)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 50)
        layer.close()
        return best

    t, u = us(412), us(448)
    assert t < 1.1 * u, (t, u)
