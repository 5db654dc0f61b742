"""The corrected CG at the sizes where its on-chip form changes shape: units of 64 columns x 4, 8, 16 or 28 rows (odd
widths, partial units, one block, one cluster, the grid) and the streamed forms that take over beyond the chip.

Tolerance: at a certified relative gap of 1e-8 the energy is within 1e-8 E of the optimum, and with A >= I that bounds
|u - u*|^2 by 2e-8 E; test_cg's 1e-4 per pixel is the bound the other CG tests use for it.
"""
import numpy as np
import pytest

import pyoracle

SHAPES = [(2, 2), (5, 3), (28, 64), (29, 65), (27, 63), (4, 200), (130, 257), (512, 128), (483, 640), (1030, 1024),
          (1001, 1101), (1001, 1104)]


def problem(H, W):
    rng = np.random.default_rng(H * 4099 + W)
    return (rng.normal(0, 0.05, (H, W)).astype(np.float32), rng.normal(0, 0.05, (H, W)).astype(np.float32),
            rng.uniform(0, 1, (3, H, W)).astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", SHAPES)
def test_cg_matches_oracle(ctx, H, W):
    gx, gy, U = problem(H, W)
    out, it, gap = ctx.stage_cg(gx, gy, U, False, 500, 1e-8)
    ref, rit, _ = pyoracle.stage_cg(gx, gy, U, False, 500, 1e-8, prec=0)
    assert abs(it - rit) <= 1 and 0 <= gap <= 1e-8
    assert np.max(np.abs(out - ref)) < 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(40, 70), (300, 200)])
def test_cg_runs_past_convergence(ctx, H, W):
    """With no gap to stop at, steps past FP32's floor leave the solution where it is."""
    gx, gy, U = problem(H, W)
    out, it, _ = ctx.stage_cg(gx, gy, U, False, 120, 0.0)
    ref, _, _ = pyoracle.stage_cg(gx, gy, U, False, 60, 0.0, prec=0)
    assert it == 120 and np.max(np.abs(out - ref)) < 1e-4
