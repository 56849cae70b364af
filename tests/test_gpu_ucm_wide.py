"""The contour map's labelling at the borders of the 512-cell segments that a
row's runs are found in (an image of 256 columns is one segment of the doubled
grid): planes with long flat stretches, so that runs cross the borders, against
the oracle's regions and strengths."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import ucm_oracle as uo  # noqa: E402


@pytest.mark.parametrize("H,W", [(2, 255), (3, 256), (5, 257), (2, 513), (9, 1100)])
def test_regions_across_segments(H, W):
    import gpb
    rng = np.random.default_rng(H * W)
    planes = np.zeros((8, H, W), np.float32)
    for x in rng.integers(0, W, max(2, W // 90)):  # a few walls, the rest flat
        planes[rng.integers(0, 8), :, x] = rng.uniform(0.2, 1.0)
    planes += np.float32(0.01) * (rng.random((8, H, W)) < 0.02)
    ctx = gpb.Context()
    u2, _ = ctx.ucm(planes, double_size=True)
    painted, w2, regions = (ctx.ucm_fetch(k) for k in (gpb.UCM_WSWT, gpb.UCM_WSWT2, gpb.UCM_REGIONS))
    ctx.close()
    want2, want, _, _ = uo.super_clean(painted.astype(np.float64))
    assert np.array_equal(w2.astype(np.float64), want2)
    assert np.array_equal(regions, want)
    assert np.abs(u2 - uo.normalize(uo.mean_pb(want2, want))).max() <= 1e-12
