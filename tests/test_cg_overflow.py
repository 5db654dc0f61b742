"""The corrected CG where the residual's square overflows FP32: the channel is not a number everywhere and the gap 1e300, so
the failure shows; the other channels are solved. (A pixel that is not a number itself stays local, as its sums say nothing.)
"""
import numpy as np
import pytest

import pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("pixels", [(1e30,), (1e30, 3e30)])  # the second: r . A r is infinity less infinity
@pytest.mark.parametrize("H,W", [(40, 70), (300, 200), (1008, 1024)])
def test_overflow_shows(ctx, H, W, pixels):
    rng = np.random.default_rng(H)
    gx, gy = (rng.normal(0, 0.05, (H, W)).astype(np.float32) for _ in range(2))
    U = rng.uniform(0, 1, (3, H, W)).astype(np.float32)
    ref, _, _ = pyoracle.stage_cg(gx, gy, U, False, 30, 0.0, prec=0)
    U[1, H // 2, W // 3:W // 3 + len(pixels)] = pixels
    out, it, gap = ctx.stage_cg(gx, gy, U, False, 30, 1e-6)
    assert it == 30 and gap == 1e300
    assert np.all(np.isnan(out[1]))
    assert np.max(np.abs(out[[0, 2]] - ref[[0, 2]])) < 1e-4
