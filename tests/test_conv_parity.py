"""The data gradient of stride-2 layers by the parity of the input pixel: patches of one row and of several, one patch and
many, channel blocks of 64 to 256, and the shapes beside them that stay with the gather kernel (a patch higher than the
image, rows that do not tile, 32 channels, 1 x 1). Tolerance: that of test_conv_matches_oracle, an FP32 sum of exact
products.
"""
import numpy as np
import pytest

import warmstart_oracle as wo

CASES = [
    # Cin, Cout, ks, batch, H, W
    (32, 64, 3, 1, 16, 32), (32, 64, 3, 2, 4, 256), (16, 64, 3, 1, 2, 512), (64, 128, 3, 1, 32, 16), (256, 256, 3, 3, 32, 16),
    (128, 128, 3, 1, 64, 8), (32, 64, 3, 1, 16, 16), (32, 64, 3, 1, 8, 96), (64, 32, 3, 1, 16, 32), (64, 64, 1, 1, 16, 32),
]


@pytest.mark.gpu
@pytest.mark.parametrize("Cin,Cout,ks,B,H,W", CASES)
def test_stride_two_data_gradient(ctx, Cin, Cout, ks, B, H, W):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(Cin * 7 + Cout + H * 1000 + W)
    w = rng.normal(0, 0.2, size=(Cout, ks * ks, Cin)).astype(np.float32)
    wq = wo.bf16(w)
    dy = wo.bf16(rng.normal(size=(B, H // 2, W // 2, Cout)))
    ref = wo.conv_dgrad(dy, wq, (B, H, W, Cin), ks, 2)
    bound = wo.conv_dgrad(np.abs(dy), np.abs(wq), (B, H, W, Cin), ks, 2)
    ddy = torch.from_numpy(np.ascontiguousarray(dy, np.float32)).cuda().to(torch.bfloat16).contiguous()
    dw = torch.from_numpy(w).cuda()
    out = torch.full((B, H, W, Cin), float("nan"), dtype=torch.float32, device="cuda")
    x = torch.zeros((B, H, W, Cin), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ctx.conv_bf16_dev(1, B, H, W, Cin, Cout, ks, 2, x.data_ptr(), ddy.data_ptr(), dw.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    err = np.abs(out.cpu().numpy().astype(np.float64) - ref)
    assert np.all(err <= 1e-5 * bound + 1e-6)
