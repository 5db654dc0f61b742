"""Branches of the warp stage and the weights that depend on the call: the warps that k_tau stores for a render (tau
alone), for IBR_color (tau and dtau/dz) and for the export, the four-pixel weights at row widths of a multiple of four
against the general kernel's other widths, views of one, two and three mask words, and quads whose boxes go to the queue
of large ones.

Renders against the FP64 oracle on the GPU's own exported warps: 1e-4, as test_render_view holds them to.
"""
import numpy as np
import pytest

import lfrv
import pyoracle


def field(V, w, h, dsf, bump):
    """V views beside each other of a plane at depth 1.5 (and, with bump, a steep ridge whose quads cover hundreds of
    target pixels)."""
    rng = np.random.default_rng(V * 31 + w)
    f = 300.0 * w / 256.0
    views = rng.uniform(0, 1, (V, 3, h, w)).astype(np.float32)
    depth = np.zeros((V, 3, h, w), np.float32)
    depth[:, 0] = 1.5
    if bump:
        depth[:, 0, h // 3:h // 3 + 2, 4:w - 4] = 1.2
        depth[:, 1, h // 3:h // 3 + 2, 4:w - 4:5] = 0.9
        depth[:, 2, h // 3:h // 3 + 2, 6:w - 4:7] = 0.8

    def camera(fx, W, H, cx):
        c = lfrv.Camera()
        for i, v in enumerate((fx, 0, 0.5 * W, 0, fx, 0.5 * H, 0, 0, 1)):
            c.K[i] = v
        for i in range(9):
            c.R[i] = 1.0 if i % 4 == 0 else 0.0
        c.t[0] = -cx
        c.width, c.height = W, H
        return c

    cams = [camera(f, w, h, 0.004 * (v - V / 2 + 0.3)) for v in range(V)]
    return views, depth, cams, camera(f * dsf, w * dsf, h * dsf, 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("bump", [False, True])
@pytest.mark.parametrize("V,w,h,dsf", [(3, 40, 24, 2), (5, 37, 21, 1), (64, 16, 12, 2), (65, 16, 12, 1), (130, 12, 10, 2)])
def test_render_equals_solve_on_exported_warps(ctx, V, w, h, dsf, bump):
    import torch

    views, depth, cams, target = field(V, w, h, dsf, bump)
    tau, dpart, zbuf = ctx.warp(depth, cams, target)
    rtau, rdpart, rzbuf = pyoracle.warp(depth, cams, target)
    # the rasterised depth: the same centre depth wherever a pixel is covered, up to pixels on a quad's edge
    assert np.mean(np.abs(zbuf - rzbuf) > 1e-3) < 0.02
    same = (tau[:, 0] < 0) == (rtau[:, 0] < 0)
    assert np.mean(same) > 0.98 and np.max(np.abs(dpart - rdpart)) < 1e-2
    assert np.max(np.abs(tau - rtau)[:, :2][np.repeat(same[:, None], 2, 1)]) < 1e-3
    cfg = lfrv.default_config(w=w, h=h, dsf=dsf, nviews=V, nchannels=3, sigma_sensor=0.01, lambda_=0.05, faithful=0,
                              cg_gap_tol=1e-6)
    dv, dd = torch.from_numpy(views).cuda(), torch.from_numpy(depth).cuda()
    out = torch.empty((3, h * dsf, w * dsf), device="cuda")
    torch.cuda.synchronize()
    ctx.render_view_dev(cfg, 1, dv.data_ptr(), dd.data_ptr(), cams, target, out.data_ptr())
    torch.cuda.synchronize()
    # ibr_gradient takes dtau/dz and so the general weights: the same image from the same warps
    got, _ = ctx.ibr_gradient(cfg, views, tau, dpart)
    assert np.max(np.abs(out.cpu().numpy() - got)) < 1e-6
    ref, _ = pyoracle.ibr_gradient(cfg, views, tau, dpart, prec=0)
    assert np.max(np.abs(got - ref)) < 1e-4
