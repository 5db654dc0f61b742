"""With per-kernel profiling on, a call's kernels run one after another, so their event times add up to no more than the
device time of the whole call: here a training step, whose weight gradients otherwise run beside the data gradients."""
import pytest

import lfrv


@pytest.mark.gpu
def test_kernel_times_fit_the_call():
    import torch

    b, h, w = 16, 256, 256
    x = torch.randn((b, h, w, 48), device="cuda").to(torch.bfloat16)
    u0, target = torch.rand((b, 3, h, w), device="cuda"), torch.rand((b, 3, h, w), device="cuda")
    stream = torch.cuda.Stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with lfrv.Context(0, stream.cuda_stream) as ctx:
        net = lfrv.WarmStart(ctx, seed=1)
        try:
            torch.cuda.synchronize()
            for k in range(3):
                if k == 2:
                    ctx.profile_enable(True)
                    e0.record(stream)
                net.train_step_dev(b, h, w, x.data_ptr(), u0.data_ptr(), target.data_ptr(), 1e-4)
            e1.record(stream)
            torch.cuda.synchronize()
            kernels = sum(ms for ms, _ in ctx.profile().values())
        finally:
            net.close()
    assert 0 < kernels <= e0.elapsed_time(e1)
