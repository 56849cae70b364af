"""The colour bins of every 24-bit colour (FP32 with an FP64 decision near bin
edges) and the texton labels with each split of a tile's groups, against the
oracle: whole numbers, equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _static(torch, ctx, packed):
    h, w = packed.shape
    src = torch.from_numpy(np.ascontiguousarray(packed, np.uint32).view(np.int32)).cuda()
    dst = torch.empty((h, w), dtype=torch.int32, device="cuda")
    ctx.texton_labels_static(w, h, src.data_ptr(), dst.data_ptr(), torch.cuda.current_stream().cuda_stream or 1)
    torch.cuda.synchronize()
    return dst.cpu().numpy().view(np.uint32)


def test_lab_bins_of_every_colour(orc):
    torch = pytest.importorskip("torch")
    import gpb
    cb = np.zeros((13, 1), np.float32)
    ctx = gpb.Context(cb)
    for part in range(16):
        packed = (np.arange(1 << 20, dtype=np.uint32) + (part << 20)).reshape(1024, 1024)
        img = np.stack([(packed >> 16) & 255, (packed >> 8) & 255, packed & 255], -1).astype(np.uint8)  # B, G, R
        want = orc.lab_bins(img).astype(np.uint32)
        got = _static(torch, ctx, packed)
        for c in range(3):
            assert np.array_equal((got >> (8 * c)) & 255, want[c]), (part, c)
    ctx.close()


@pytest.mark.parametrize("H,W", [(32, 32), (33, 130), (272, 300), (740, 730)])  # splits 4, 4, 2, 1
def test_texton_labels_with_each_split(orc, H, W):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import synth
    img = synth.voronoi_image(H, W, 20, 8.0, synth.SEED_BASE + 171 + W)
    cb = synth.make_codebook(img, synth.SEED_BASE + 171 + W, n_sample=1024)
    ctx = gpb.Context(cb)
    got = _static(torch, ctx, synth.pack_bgr(img)) >> 24
    ctx.close()
    assert np.array_equal(got, orc.texton_map(orc.grey_bgr(img), cb))
