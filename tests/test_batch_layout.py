"""Batched targets of odd pixel counts: where their buffers lie in the pool, and that each gives what it gives alone.

Tolerances are test_batch's (the batched CG sums the dot products over another block partition): equal iteration counts,
the gap to 1e-6 relative, 1e-5 per pixel), for seeded targets test_warmstart's (60 dB, one iteration).
"""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import lfrv
from scenes import gradient_config

CSRC = Path(__file__).resolve().parents[1] / "light-field-remote-vision_gb300" / "csrc"

SRC = r"""
#include <cstdio>
#include "batch_layout.h"
using namespace lfrv;
int main() {
    long bad = 0, n = 0;
    for (size_t w = 2; w < 320; ++w)
        for (size_t h = 2; h < 48; ++h)
            for (int seeded = 0; seeded < 2; ++seeded) {
                const size_t N = w * h, lens[8] = {3 * N, N, N, 3 * N, 3 * N, 16, 3 * N, 24 * N};
                const BatchLayout L = batch_layout(N, seeded != 0, 48);
                const size_t offs[8] = {L.U, L.gx, L.gy, L.dA, L.dB, L.state, L.seed, L.input};
                size_t end = 0;
                for (int i = 0; i < (seeded ? 8 : 6); ++i) {
                    bad += (offs[i] * 4) % 16 != 0 || offs[i] < end;  // in order, without overlap
                    end = offs[i] + lens[i];
                }
                bad += (L.size * 4) % 16 != 0 || L.size < end;  // the next target
                ++n;
            }
    float f[4];
    float *p = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(f) + 7) & ~(uintptr_t)7);
    bad += !cg_borders_aligned(p, p) || cg_borders_aligned(p, p + 1) || cg_borders_aligned(p + 1, p);
    std::printf("%ld %ld\n", bad, n);
    return 0;
}
"""


def test_sections_are_aligned(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(SRC)
    subprocess.run([cc, "-std=c++17", "-O1", f"-I{CSRC}", "-o", str(exe), str(src)], check=True)
    bad, n = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert n > 20000 and bad == 0


def job(torch, preset, w, h, seed=1, **kw):
    sc = lfrv.synth_scene(lfrv.scene_params(preset, w=w, h=h, seed=seed, **kw))
    cfg = gradient_config(sc)
    keep = [torch.from_numpy(sc.views).cuda(), torch.from_numpy(sc.depth).cuda(),
            torch.zeros((3, cfg.h * cfg.dsf, cfg.w * cfg.dsf), device="cuda")]
    return keep, dict(cfg=cfg, algorithm=1, d_views=keep[0].data_ptr(), d_depth=keep[1].data_ptr(), cams=sc.cams,
                      target=sc.target, d_out=keep[2].data_ptr())


BATCHES = [
    [(1, 65, 65, {})],
    [(1, 201, 133, {}), (1, 65, 33, {}), (1, 48, 48, {}), (1, 75, 51, {})],
    [(1, 27, 21, dict(dsf=3)), (2, 40, 36, {})],
    [(1, 1001, 541, {}), (1, 65, 65, {})],                        # the first needs more than half of the blocks
    [(1, 513 - 2 * k, 415, {}) for k in range(5)],                 # more than one launch holds
    [(1, 3, 401, {}), (1, 33, 65, {})],                            # the first is too thin for the on-chip form
]


@pytest.mark.gpu
@pytest.mark.parametrize("specs", BATCHES)
def test_odd_targets_match_single(ctx, specs):
    import torch

    made = [job(torch, p, w, h, seed=k + 3, **kw) for k, (p, w, h, kw) in enumerate(specs)]
    torch.cuda.synchronize()
    stats = ctx.render_views_dev([j for _, j in made])
    torch.cuda.synchronize()
    for (keep, j), st in zip(made, stats):
        got = keep[2].cpu().numpy().copy()
        st1 = ctx.render_view_dev(j["cfg"], 1, j["d_views"], j["d_depth"], j["cams"], j["target"], j["d_out"])
        torch.cuda.synchronize()
        assert st.outer_iterations == st1.outer_iterations
        assert st.hole_fill_iterations == st1.hole_fill_iterations
        assert abs(st.gap - st1.gap) <= 1e-6 * max(st1.gap, 1e-12) + 1e-9
        assert np.max(np.abs(got - keep[2].cpu().numpy())) < 1e-5


@pytest.mark.gpu
def test_odd_targets_from_host_buffers(ctx):
    import torch

    made = [job(torch, 1, w, h, seed=k + 11) for k, (w, h) in enumerate([(65, 33), (75, 51), (48, 40)])]
    ctx.render_views_dev([j for _, j in made])
    torch.cuda.synchronize()
    host = [[t.cpu() for t in keep] for keep, _ in made]
    jobs = []
    for (views, depth, out), (_, j) in zip(host, made):
        out.zero_()
        jobs.append(dict(j, d_views=views.data_ptr(), d_depth=depth.data_ptr(), d_out=out.data_ptr()))
    ctx.render_views(jobs)
    for (_, _, out), (keep, _) in zip(host, made):
        np.testing.assert_array_equal(out.numpy(), keep[2].cpu().numpy())


@pytest.mark.gpu
def test_seeded_target_after_odd_ones(ctx):
    """A target seeded by the warm start behind targets of odd pixel counts (which run unseeded)."""
    import torch

    made = [job(torch, 1, w, h, seed=k + 20) for k, (w, h) in enumerate([(65, 33), (64, 64), (75, 51), (128, 40)])]
    net = lfrv.WarmStart(ctx, seed=5)
    try:
        torch.cuda.synchronize()
        stats = ctx.render_views_dev([j for _, j in made], net)
        torch.cuda.synchronize()
        for (keep, j), st in zip(made, stats):
            got = keep[2].cpu().numpy().copy()
            if j["cfg"].w % 8 == 0:
                st1 = net.render_view_dev(j["cfg"], j["d_views"], j["d_depth"], j["cams"], j["target"], j["d_out"])
            else:
                st1 = ctx.render_view_dev(j["cfg"], 1, j["d_views"], j["d_depth"], j["cams"], j["target"], j["d_out"])
            torch.cuda.synchronize()
            assert abs(st.outer_iterations - st1.outer_iterations) <= 1 and st.gap <= 1e-6
            assert lfrv.psnr(got, keep[2].cpu().numpy()) > 60.0
    finally:
        net.close()
