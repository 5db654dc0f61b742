"""The persistent ROF where values leave FP32's finite range: an infinity, a not-a-number or a number whose square
overflows, inside the image and in the last column, row and corner. It has to spread as in the reference's loop (a
difference that does not exist adds nothing, a dual of infinite norm is scaled by r / inf = 0, an infinite numerator
divided stays infinite): not-a-number, infinite and finite values at the same places as in the FP32 restatement of that
loop, and the finite ones within test_rof_vs_fp64's 1e-5, relative beyond 1.
"""
import numpy as np
import pytest

import pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("niter", [1, 2, 5])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e25, 3e38])
@pytest.mark.parametrize("H,W", [(1, 1), (40, 70), (300, 200)])
def test_rof_nonfinite(ctx, H, W, value, niter):
    rng = np.random.default_rng(H * 1000 + W)
    F = rng.uniform(0, 1, (3, H, W)).astype(np.float32)
    g = rng.uniform(0.05, 5, (H, W)).astype(np.float32)
    P = rng.normal(0, 0.5, (6, H, W)).astype(np.float32)
    U = F.copy()
    U[0, H // 2, W - 1] = U[1, H - 1, W // 2] = U[2, H // 3, W // 3] = U[0, H - 1, W - 1] = value
    F[1, 0, 0] = value
    tau = sigma = np.float32(0.3 / np.sqrt(8.0))
    with np.errstate(all="ignore"):
        got = ctx.stage_rof(niter, tau, sigma, 0.05, F, g, U.copy(), P)
        ref = pyoracle.stage_rof(niter, tau, sigma, 0.05, F, g, U.copy(), P, prec=1)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        np.testing.assert_array_equal(np.isinf(a), np.isinf(b))
        ok = np.isfinite(b)
        assert np.all(a[~ok & ~np.isnan(b)] == b[~ok & ~np.isnan(b)])
        err = np.abs(a[ok].astype(np.float64) - b[ok]) / np.maximum(np.abs(b[ok]), 1.0)
        assert err.max(initial=0.0) < 1e-5
