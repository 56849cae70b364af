"""The plain eigensolver's two forms of a step -- three launches for batches of
many 2048-pixel tiles, five for few -- at the edges of a tile: an image alone
against copies of it that pass the line of 96 tiles.  Every sum belongs to one
patch and runs in the same order in both, so the outputs are equal to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(32, 32), (32, 64), (32, 65), (43, 143)])
def test_few_tiles_equal_many(h, w):
    import gpb
    from gpb import synth
    img = synth.voronoi_image(h, w, 8, 8.0, synth.SEED_BASE + 163)
    cb = synth.make_codebook(synth.voronoi_image(96, 96, 12, 8.0, synth.SEED_BASE + 163), synth.SEED_BASE + 163,
                             n_sample=1024)
    px = synth.pack_bgr(img)
    ctx = gpb.Context(cb, eig_mode=gpb.EIG_LANCZOS, keep_intermediates=1)
    n = 96 // -(-h * w // 2048) + 1
    many = ctx.compute_batch([px] * n)
    X = [ctx.fetch(k, n - 1, s, np.float32) for k, s in (("evals", (9,)), ("evecs", (9, h * w)))]
    one = ctx.compute_batch([px])[0]
    for got, want in zip([ctx.fetch("evals", 0, (9,), np.float32), ctx.fetch("evecs", 0, (9, h * w), np.float32)], X):
        assert np.array_equal(got, want)
    for m in (many[0], many[-1]):
        assert np.array_equal(one[0], m[0]) and np.array_equal(one[1], m[1])
    ctx.close()
