"""The gathers through the inverse map at every footprint (dsf 1 to 4: four entries ahead up to three taps a side, one by
one beyond), and the z-buffer's queues at quads around their lines (3 x 3 centres: unrolled; up to 512: a warp; more:
sixteen warps), against the FP64 oracle with test_ibr_color_vs_fp64's 1e-4 and test_warp_stage_paths' depth bounds.
"""
import numpy as np
import pytest

import lfrv
import pyoracle
from scenes import color_config, rel_err
from test_warp_stage_paths import field


@pytest.mark.gpu
@pytest.mark.parametrize("dsf", [1, 2, 3, 4])
@pytest.mark.parametrize("kw", [dict(faithful=1, niter=4, dt_beta=0.5, gw_type=1, gradient_step=0.25),
                                dict(faithful=0, niter=3, cg_gap_tol=0.0)])
def test_gathers(ctx, dsf, kw):
    sc = lfrv.synth_scene(lfrv.scene_params(1, w=27, h=21, seed=dsf, dsf=dsf))
    tau, dpart, _ = (np.float32(a) for a in pyoracle.warp(sc.depth, sc.cams, sc.target))
    cfg = color_config(sc, **kw)
    out, _ = ctx.ibr_color(cfg, sc.views, tau, dpart)
    ref, _ = pyoracle.ibr_color(cfg, sc.views, tau, dpart, prec=0)
    assert rel_err(out, ref) <= 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("side", [2.5, 4, 9.5, 10.5, 22, 23, 40])
@pytest.mark.parametrize("tilt", [0.0, 0.3])
def test_quads_of_many_pixels(ctx, side, tilt):
    views, depth, cams, target = field(3, 24, 20, 1, False)
    depth[:, 1:] = tilt
    W, H = 120, 90
    target.K[0] = target.K[4] = target.K[0] * side
    target.K[2], target.K[5] = 0.5 * W, 0.5 * H
    target.width, target.height = W, H
    tau, _, zbuf = ctx.warp(depth, cams, target)
    rtau, _, rzbuf = pyoracle.warp(depth, cams, target)
    assert np.mean(np.abs(zbuf - rzbuf) > 1e-3) < 0.02
    assert np.mean((tau[:, 0] < 0) == (rtau[:, 0] < 0)) > 0.98
