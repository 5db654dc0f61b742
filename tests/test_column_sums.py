"""Bias gradients (column sums of the output gradients) and the reduction of the weight gradient's splits, at pixel counts
with remainders: fewer pixels than a block's lanes, one split, splits that do not divide by the lanes.

The loss is mean((u0 + y - t)^2) with the untrained output layer (y = 0), so the output bias gradient is the column sum of
2 (u0 - t) / (3 P) rounded to BF16, up to the order of an FP32 sum of P terms: sqrt(P) 2^-24 of the terms' magnitude is the
expected size, 64 of those the bound.
"""
import numpy as np
import pytest

import lfrv
import warmstart_oracle as wo


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,W", [(1, 8, 8), (1, 8, 24), (3, 8, 16), (1, 40, 56), (2, 104, 72), (1, 256, 200)])
def test_output_bias_gradient_is_the_column_sum(ctx, B, H, W):
    torch = pytest.importorskip("torch")
    net = lfrv.WarmStart(ctx, seed=3)
    rng = np.random.default_rng(H * 1000 + W)
    x = torch.from_numpy(rng.normal(size=(B, H, W, 48)).astype(np.float32)).cuda().to(torch.bfloat16).contiguous()
    u0 = torch.from_numpy(rng.uniform(0, 1, (B, 3, H, W)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.uniform(0, 1, (B, 3, H, W)).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    _, g = net.gradients_dev(B, H, W, x.data_ptr(), u0.data_ptr(), t.data_ptr())
    net.close()
    P = B * H * W
    scale = np.float32(2) / (np.float32(3) * np.float32(P))  # in FP32 as the kernel does, so that BF16 rounds alike
    dy = np.asarray(wo.bf16((u0 - t).cpu().numpy() * scale), np.float64)
    ref = dy.sum(axis=(0, 2, 3))
    bound = 64 * np.sqrt(P) * 2.0 ** -24 * np.abs(dy).max() + 1e-9
    assert np.max(np.abs(g[-3:] - ref)) < bound
