"""An SM budget keeps the other SMs free: kernels of another stream that need an SM of their own run beside a budgeted layer's
long gate/up product instead of waiting for its down product to leave."""
import pytest
import torch

from mgpt_b200 import MoELayer

pytestmark = pytest.mark.gpu


def _layer(C, H, E, k, sms):
    layer = MoELayer(C, H, E, k, mode="bf16")
    gen = torch.Generator(device="cuda").manual_seed(3)
    for p in layer.get_parameters():
        p.normal_(0.0, 0.02, generator=gen)
    layer.sync_weights()
    layer.lib.mgpt_moe_set_sm_budget(layer._h, sms)
    return layer


def test_other_streams_find_free_sms():
    total = torch.cuda.get_device_properties(0).multi_processor_count
    # gate/up takes most of the call; with down's CTAs let in early the two would hold every SM
    large, small = _layer(1024, 2816, 8, 2, total * 2 // 3), _layer(256, 256, 4, 2, total // 4)
    x, xs = (torch.randn(n, C, device="cuda").bfloat16() for n, C in ((98304, 1024), (600, 256)))
    y, ys = torch.empty_like(x), torch.empty_like(xs)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()

    def run():
        begin, end_large, end_small = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        torch.cuda.synchronize()
        begin.record(a)
        b.wait_stream(a)
        with torch.cuda.stream(a):
            large.forward_inference_into(x, y)
            end_large.record(a)
        with torch.cuda.stream(b):
            for _ in range(20):                 # some of them begin after the large layer's gate/up
                small.forward_inference_into(xs, ys)
            end_small.record(b)
        torch.cuda.synchronize()
        return begin.elapsed_time(end_small), begin.elapsed_time(end_large)

    run()
    times = [run() for _ in range(3)]
    # 20 small calls take a quarter of the large one's time; held up by down they end with it
    assert min(s / l for s, l in times) < 0.75, times
    large.check_status()
    small.check_status()
    large.close()
    small.close()
