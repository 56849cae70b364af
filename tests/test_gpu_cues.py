"""The half-disc histogram cues at the edges of the kernel's 8 x 16 pixel
tiles and of its bin counts, against the oracle: the smallest patch, sides one
past and one short of a tile, 1 and 32 codewords, and an image of two flat
colours (histograms of one or two bins).  Tolerance as in the parity tests:
cue maps 1e-5, weighted sums 1e-6 absolute (FP32 against FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# src/multiscalePb.cpp:19-26
W_MPB = [0.0146, 0.0145, 0.0163, 0.0210, 0.0243, 0.0287, 0.0166, 0.0185, 0.0204, 0.0101, 0.0111, 0.0141]


@pytest.mark.parametrize("H,W,k,sigma", [(32, 32, 32, 8.0), (33, 47, 32, 8.0), (39, 65, 1, 8.0), (41, 34, 8, 30.0),
                                         (40, 48, 2, 0.0)])
def test_cues_at_tile_and_bin_edges(orc, H, W, k, sigma):
    import gpb
    from gpb import synth
    img = synth.voronoi_image(H, W, 2 if sigma == 0 else 6, sigma, synth.SEED_BASE + 131 + W, ramp=0.0 if sigma == 0 else 40.0)
    cb = synth.make_codebook(img, synth.SEED_BASE + 131 + W, k=k, n_sample=1024)
    ref = orc.globalpb(img, cb, intermediates=True)
    ctx = gpb.Context(cb, keep_intermediates=1, eig_mode=gpb.EIG_WARM)
    ctx.compute_batch([synth.pack_bgr(img)])
    cues = ctx.fetch("cues", 0, (12, 8, H, W), np.float32)
    assert np.abs(cues - ref["cues"]).max() < 1e-5
    mpb_o = np.tensordot(W_MPB, ref["cues"], 1)
    assert np.abs(ctx.fetch("mpb_o", 0, (8, H, W), np.float32) - mpb_o).max() < 1e-6
    ctx.close()
