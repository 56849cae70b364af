"""A batch of too few tiles to time settles on the texton variant that the
static entry point takes at that size: four sets of threads per tile."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(32, 32), (64, 80), (90, 112)])  # 4, 20 and 42 tiles of 16 x 16
def test_small_batch_takes_four_sets(H, W):
    import gpb
    from gpb import synth
    img = synth.voronoi_image(H, W, 6, 8.0, synth.SEED_BASE + 203)
    ctx = gpb.Context(synth.make_codebook(img, synth.SEED_BASE + 203, k=4, n_sample=512), eig_mode=gpb.EIG_WARM)
    ctx.compute_batch([synth.pack_bgr(img)])
    chosen = [v[0] for k, v in ctx.tuning_report().items() if k.startswith("texton/")]
    ctx.close()
    assert chosen == [2]
