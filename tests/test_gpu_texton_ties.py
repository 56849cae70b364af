"""Texton labels where every pixel is decided in FP64: each codeword of the
codebook is there twice, so the two nearest are always equally far and the
first of them wins.  More pixels than the repair launch has CTAs (1216), and
fewer.  Whole numbers, equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(32, 33), (33, 38), (64, 80)])
def test_labels_with_every_pixel_tied(orc, H, W):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import synth
    img = synth.voronoi_image(H, W, 8, 8.0, synth.SEED_BASE + 181)
    cb = np.repeat(synth.make_codebook(img, synth.SEED_BASE + 181, k=11, n_sample=1024), 2, 1)
    src = torch.from_numpy(synth.pack_bgr(img).view(np.int32)).cuda()
    dst = torch.empty((H, W), dtype=torch.int32, device="cuda")
    ctx = gpb.Context(np.ascontiguousarray(cb))
    ctx.texton_labels_static(W, H, src.data_ptr(), dst.data_ptr(), torch.cuda.current_stream().cuda_stream or 1)
    torch.cuda.synchronize()
    ctx.close()
    got = dst.cpu().numpy().view(np.uint32) >> 24
    assert (got % 2 == 0).all() and np.array_equal(got, orc.texton_map(orc.grey_bgr(img), cb))
