"""The decoder's fused upsampling at every patch shape of the TMA kernel (one row of 128 pixels, several rows, one patch and
many, one and several passes of 32 columns) against the gather kernel, which writes each pixel's 2 x 2 block by itself.

The two run the same sums; the bound is test_network_gradients_match_oracle's for a prediction.
"""
import numpy as np
import pytest

import lfrv
import warmstart_oracle as wo


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,W", [(2, 64, 128), (1, 128, 128), (1, 32, 256), (3, 256, 64), (1, 16, 512), (1, 8, 1024), (1, 16, 2048)])
def test_upsampling_layers_match_the_gather_kernel(ctx, B, H, W):
    torch = pytest.importorskip("torch")
    net = lfrv.WarmStart(ctx, seed=3)
    net.set_params(wo.init_params(3))
    rng = np.random.default_rng(H + W)
    x = torch.from_numpy(rng.random((B, H, W, 48)).astype(np.float32)).cuda().to(torch.bfloat16).contiguous()
    u0 = torch.from_numpy(rng.random((B, 3, H, W)).astype(np.float32)).cuda()
    pred = [torch.full((B, 3, H, W), float("nan"), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    try:
        for p, which in zip(pred, (0, 2)):
            lfrv.set_conv_kernel(which)
            net.forward_dev(B, H, W, x.data_ptr(), u0.data_ptr(), p.data_ptr())
            torch.cuda.synchronize()
    finally:
        lfrv.set_conv_kernel(0)
    net.close()
    y = (pred[1] - u0).abs().max().item()
    assert y > 0 and (pred[0] - pred[1]).abs().max().item() < 2e-2 * max(1.0, y)
