"""Inverse map buckets that hold several source pixels of one view: their entries arrive in any order and are sorted, so
the gathers sum in a fixed order. The warps shrink the views by 1 / scale, which puts about 8 scale^-2 entries into a
bucket: 8 (no sort), 18, 50, 128, 512 (past the shared-memory sort) and all 6144 at once.

Weighted averages of [0, 1] values against the FP64 oracle: 1e-4, the bound of the other gather tests.
"""
import numpy as np
import pytest

import lfrv
import pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("dsf", [1, 2])
@pytest.mark.parametrize("scale", [1.0, 0.67, 0.4, 0.25, 0.125, 0.0])
def test_shrunken_views(ctx, scale, dsf):
    rng = np.random.default_rng(3)
    V, h, w = 8, 24, 32
    y, x = np.mgrid[0:h, 0:w] + 0.5
    tau = np.zeros((V, 3, h, w), np.float32)
    for v in range(V):
        tau[v, 0] = dsf * (8.3 + 0.11 * v + scale * x)
        tau[v, 1] = dsf * (7.2 - 0.07 * v + scale * y)
    dpart = np.zeros((V, 3, h, w), np.float32)
    views = rng.uniform(0, 1, (V, 3, h, w)).astype(np.float32)
    cfg = lfrv.default_config(w=w, h=h, dsf=dsf, nviews=V, nchannels=3, sigma_sensor=0.01, lambda_=0.05, faithful=0,
                              cg_gap_tol=1e-6)
    out, _ = ctx.ibr_gradient(cfg, views, tau, dpart)
    again, _ = ctx.ibr_gradient(cfg, views, tau, dpart)
    np.testing.assert_array_equal(out, again)
    ref, _ = pyoracle.ibr_gradient(cfg, views, tau, dpart, prec=0)
    assert np.max(np.abs(out - ref)) < 1e-4
