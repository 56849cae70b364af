"""gpb_stitch_device with more patches than one pass over the boxes takes (256),
several of them over the same tile, an image that is no multiple of the tile
and boxes that leave it, against the same stitching on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_stitch_many_overlapping_patches(mode):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import synth
    rng = np.random.default_rng(5)
    img = synth.voronoi_image(128, 160, 12, 8.0, synth.SEED_BASE + 191)
    cb = synth.make_codebook(img, synth.SEED_BASE + 191, k=4, n_sample=512)
    sizes = [(32, 32), (33, 40), (47, 35)]
    shapes = [sizes[i % 3] for i in range(270)]
    packed = synth.pack_bgr(img)
    ctx = gpb.Context(cb, eig_mode=gpb.EIG_WARM)
    outs = ctx.compute_batch([np.ascontiguousarray(packed[i % 60:i % 60 + h, i % 90:i % 90 + w])
                              for i, (h, w) in enumerate(shapes)])
    H, W = 77, 101
    places = []
    for h, w in shapes:
        ix, iy = int(rng.integers(0, 6)), int(rng.integers(0, 6))
        places.append((int(rng.integers(-20, W - 10)), int(rng.integers(-20, H - 10)), ix, iy, w - ix - 2, h - iy - 3))
    d_nm = torch.full((H, W), -7.0, device="cuda")
    d_or = torch.full((8, H, W), -7.0, device="cuda")
    ctx.stitch_device(mode, W, H, places, d_nm.data_ptr(), d_or.data_ptr(), ramp=4)
    ctx.close()
    want = np.full((9, H, W), -7.0)
    acc = np.zeros((10, H, W))
    for (nm, orr), (h, w), (x0, y0, ix, iy, iw, ih) in zip(outs, shapes, places):
        v = np.concatenate([nm.reshape(1, h, w), orr.reshape(8, h, w)])
        if mode != 1:
            ix, iy, iw, ih = 0, 0, w, h
        ya, yb, xa, xb = max(0, y0 + iy), min(H, y0 + iy + ih), max(0, x0 + ix), min(W, x0 + ix + iw)
        if yb <= ya or xb <= xa:
            continue
        src = v[:, ya - y0:yb - y0, xa - x0:xb - x0]
        if mode == 2:
            yy, xx = np.meshgrid(np.arange(ya - y0, yb - y0) + 0.5, np.arange(xa - x0, xb - x0) + 0.5, indexing="ij")
            wt = np.ones_like(yy)
            for cond, dist in ((y0 > 0, yy), (x0 > 0, xx), (y0 + h < H, h - yy), (x0 + w < W, w - xx)):
                if cond:
                    wt = np.minimum(wt, dist / 4.0)
            acc[0, ya:yb, xa:xb] += wt
            acc[1:, ya:yb, xa:xb] += wt * src
        else:
            want[:, ya:yb, xa:xb] = src
    got = np.concatenate([d_nm.cpu().numpy()[None], d_or.cpu().numpy()])
    if mode == 2:
        want = np.where(acc[0] > 0, acc[1:] / np.where(acc[0] > 0, acc[0], 1), -7.0)
        assert np.abs(got - want).max() < 1e-5  # FP32 sums of up to 40 weighted values in [0, 1]
    else:
        assert np.array_equal(got, want.astype(np.float32))


@pytest.mark.parametrize("n,H,W", [(1, 2 ** 21 + 40, 1), (128, 70, 90), (129, 70, 90)])
def test_stitch_box_counts_and_tall_image(n, H, W):
    """Around the 128 boxes that travel in the launch, and an image of more
    rows of tiles than a grid's second dimension holds: copies, so exact."""
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import synth
    img = synth.voronoi_image(64, 64, 12, 8.0, synth.SEED_BASE + 193)
    cb = synth.make_codebook(img, synth.SEED_BASE + 193, k=4, n_sample=512)
    packed = synth.pack_bgr(img)
    ctx = gpb.Context(cb, eig_mode=gpb.EIG_WARM)
    outs = ctx.compute_batch([np.ascontiguousarray(packed[i % 30:i % 30 + 32, i % 29:i % 29 + 32]) for i in range(n)])
    places = [(7 * i % W, H - 35 - 11 * i % (H - 34), 0, 0, 32, 32) for i in range(n)]
    d_nm = torch.full((H, W), -7.0, device="cuda")
    d_or = torch.full((8, H, W), -7.0, device="cuda")
    ctx.stitch_device(gpb.STITCH_LAST, W, H, places, d_nm.data_ptr(), d_or.data_ptr())
    ctx.close()
    want = np.full((9, H, W), -7.0, np.float32)
    for (nm, orr), (x0, y0, *_) in zip(outs, places):
        v = np.concatenate([nm.reshape(1, 32, 32), orr.reshape(8, 32, 32)])
        want[:, y0:y0 + 32, x0:x0 + 32] = v[:, :min(32, H - y0), :min(32, W - x0)]
    assert np.array_equal(d_nm.cpu().numpy(), want[0]) and np.array_equal(d_or.cpu().numpy(), want[1:])
