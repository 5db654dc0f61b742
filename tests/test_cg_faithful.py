"""The reference's five CG iterations (faithful) in one launch: images of a part of a block, ragged rows, several blocks
and more pixels than resident threads.

Tolerance: test_cg's 1e-4 per pixel, the bound the other CG tests use (the iterates differ by the order of the sums).
"""
import numpy as np
import pytest

import pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(2, 2), (2, 300), (5, 3), (31, 17), (130, 257), (600, 701)])
def test_faithful_cg_matches_oracle(ctx, H, W):
    rng = np.random.default_rng(H * 4099 + W)
    gx, gy = (rng.normal(0, 0.05, (H, W)).astype(np.float32) for _ in range(2))
    U = rng.uniform(0, 1, (3, H, W)).astype(np.float32)
    out, it, _ = ctx.stage_cg(gx, gy, U, True, 500, 1e-8)
    ref, rit, _ = pyoracle.stage_cg(gx, gy, U, True, 500, 1e-8, prec=0)
    assert it == rit == 5
    assert np.max(np.abs(out - ref)) < 1e-4
