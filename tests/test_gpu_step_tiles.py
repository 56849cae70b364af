"""The block solvers at the edges of the block step's 16 x 16 pixel tiles (its
operator is stored tile by tile): FP64 residual of every eigenpair on the
fetched affinities, and the default against the autotuned step variant to the
bit.  Tolerance: 3 x eig_tol, as in the parity tests."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _residual(orc, Wd, evals, evecs):
    H, W, _ = Wd.shape
    dy, dx = orc.stencil()
    pad = np.zeros((9, H + 10, W + 10))
    deg = Wd.sum(-1)
    y = evecs.reshape(9, H, W)
    pad[:, 5:-5, 5:-5] = y / np.sqrt(deg)
    Ax = y.copy()
    for k in range(81):
        sh = pad[:, 5 + dy[k]:5 + dy[k] + H, 5 + dx[k]:5 + dx[k] + W]
        Ax -= Wd[..., k] * sh / np.sqrt(deg)
    r = (Ax - evals[:, None, None] * y).reshape(9, -1)
    return (np.linalg.norm(r, axis=1) / np.linalg.norm(y.reshape(9, -1), axis=1)).max()


@pytest.mark.parametrize("mode", [1, 2])
def test_residuals_at_tile_edges(orc, mode):
    import gpb
    from gpb import synth
    sizes = [(32, 32), (33, 47), (47, 33), (48, 49), (40, 64), (49, 80)]
    img = synth.voronoi_image(120, 200, 12, 8.0, synth.SEED_BASE + 151)
    cb = synth.make_codebook(img, synth.SEED_BASE + 151, n_sample=1024)
    patches = [synth.pack_bgr(img[3 * i:3 * i + h, 5 * i:5 * i + w]) for i, (h, w) in enumerate(sizes)]
    ctx = gpb.Context(cb, keep_intermediates=1, eig_mode=mode)
    for _ in range(3):  # with the autotuner's trials, then its choice
        out = ctx.compute_batch(patches)
    for i, (h, w) in enumerate(sizes):
        Wd = ctx.fetch("W", i, (h, w, 81), np.float32).astype(np.float64)
        ev = ctx.fetch("evals", i, (9,), np.float32).astype(np.float64)
        X = ctx.fetch("evecs", i, (9, h * w), np.float32).astype(np.float64)
        assert _residual(orc, Wd, ev, X) <= 3 * ctx.params.eig_tol, (h, w)
    ctx.close()
    os.environ["GPB_NO_TUNE"] = "1"
    try:
        plain = gpb.Context(cb, eig_mode=mode)
    finally:
        del os.environ["GPB_NO_TUNE"]
    for (a, b), (c, d) in zip(out, plain.compute_batch(patches)):
        assert np.array_equal(a, c) and np.array_equal(b, d)
    plain.close()
