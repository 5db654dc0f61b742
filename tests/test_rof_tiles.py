"""The persistent ROF at the edges of its tiles (32 columns, 8, 16 or 32 rows, halos of 4 to 10 pixels) and super-steps:
images smaller than a tile, one pixel over, several tiles, and iteration counts around K.

25 iterations stay within 1e-5 of FP64 (test_rof_vs_fp64); the iteration is a contraction, so that bound holds for more.
"""
import numpy as np
import pytest

import pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("niter", [1, 7, 33])
@pytest.mark.parametrize("H,W", [(1, 1), (3, 40), (16, 32), (17, 33), (15, 31), (40, 97), (130, 70), (300, 40)])
def test_rof_vs_fp64(ctx, H, W, niter):
    rng = np.random.default_rng(H * 1000 + W)
    F = rng.uniform(0, 1, (3, H, W)).astype(np.float32)
    g = rng.uniform(0.05, 5, (H, W)).astype(np.float32)
    P = rng.normal(0, 0.5, (6, H, W)).astype(np.float32)
    tau = sigma = np.float32(0.3 / np.sqrt(8.0))
    U1, P1 = ctx.stage_rof(niter, tau, sigma, 0.05, F, g, F.copy(), P)
    rU, rP = pyoracle.stage_rof(niter, tau, sigma, 0.05, F, g, F.copy(), P, prec=0)
    assert np.max(np.abs(U1 - rU)) < 1e-5
    assert np.max(np.abs(P1 - rP)) < 1e-5
