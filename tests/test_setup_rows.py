"""The IBR_gradient set-up's anchor-row kernel at the edges of its tiles: 62 output columns per warp and 13 to 15 (two
anchor rows per warp) or 6 to 7 (one) output rows per block, footprints of 2 and 3 taps, taps cut off by every image
border, and pixels reached by one vanishing tap only. The weighted average, the gradient splat and the mask through
lfrv_stage_u_gradient are not this kernel; the whole solve with no CG step (cg_max_iter 0) is its anchor image.

Averages of [0, 1] values against the FP64 oracle: 1e-4, the bound of the other gather tests.
"""
import numpy as np
import pytest

import lfrv
import pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("dsf", [1, 2])
@pytest.mark.parametrize("w,h", [(2, 2), (31, 7), (62, 15), (63, 14), (125, 16), (350, 230)])
def test_anchor_image(ctx, w, h, dsf):
    rng = np.random.default_rng(w * 1000 + h)
    V = 5
    y, x = np.mgrid[0:h, 0:w] + 0.5
    tau = np.zeros((V, 3, h, w), np.float32)
    for v in range(V):
        s = 0.9 + 0.05 * v
        tau[v, 0] = dsf * (s * x + rng.uniform(-1, 1))
        tau[v, 1] = dsf * (s * y + rng.uniform(-1, 1))
    tau[0, 0], tau[0, 1] = dsf * x, dsf * y  # anchors on exact half pixels: vanishing taps
    dpart = np.zeros((V, 3, h, w), np.float32)
    views = rng.uniform(0, 1, (V, 3, h, w)).astype(np.float32)
    cfg = lfrv.default_config(w=w, h=h, dsf=dsf, nviews=V, nchannels=3, sigma_sensor=0.01, lambda_=0.05, faithful=0,
                              cg_gap_tol=0.0, cg_max_iter=0)
    out, _ = ctx.ibr_gradient(cfg, views, tau, dpart)
    ref, _ = pyoracle.ibr_gradient(cfg, views, tau, dpart, prec=0)
    assert np.max(np.abs(out - ref)) < 1e-4
    vis = ctx.stage_gradient_visibility(cfg, tau)
    assert vis.any()
    # one CG step brings the splatted gradient in
    cfg.cg_max_iter = 1
    out, _ = ctx.ibr_gradient(cfg, views, tau, dpart)
    ref, _ = pyoracle.ibr_gradient(cfg, views, tau, dpart, prec=0)
    assert np.max(np.abs(out - ref)) < 1e-4
