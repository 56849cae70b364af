"""gpb_stitch_device with boxes scattered over an image much larger than they
are (a CTA per tile of a box instead of one per tile around all boxes): boxes
that overlap, share tiles and leave the image, against the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 7, 140])  # 140: more boxes than travel in the launch
def test_stitch_scattered(mode, n):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import synth
    rng = np.random.default_rng(n)
    img = synth.voronoi_image(96, 96, 12, 8.0, synth.SEED_BASE + 197)
    cb = synth.make_codebook(img, synth.SEED_BASE + 197, k=4, n_sample=512)
    packed = synth.pack_bgr(img)
    shapes = [[(32, 32), (33, 40), (47, 35)][i % 3] for i in range(n)]
    ctx = gpb.Context(cb, eig_mode=gpb.EIG_WARM)
    outs = ctx.compute_batch([np.ascontiguousarray(packed[i % 40:i % 40 + h, i % 50:i % 50 + w])
                              for i, (h, w) in enumerate(shapes)])
    H, W = 1500, 2001
    at = [(int(rng.integers(-30, W)), int(rng.integers(-30, H))) for _ in range(n)]
    for i in range(2, n, 3):  # beside, over and away from the box before
        at[i] = (at[i - 1][0] + int(rng.integers(-40, 40)), at[i - 1][1] + int(rng.integers(-40, 40)))
    places = [[x0, y0, 2, 1, w - 5, h - 3] for (h, w), (x0, y0) in zip(shapes, at)]
    if n > 1:  # earlier boxes that touch a tile only outside the image, or not at all, do not own it
        places[1][:2], places[3][:2] = (W + 4, 45), (W - 25, 40)
        places[4][:], places[5][:2] = [700, 600, 3, 3, 0, 9], (690, 595)
    at = [tuple(p[:2]) for p in places]
    places = [tuple(p) for p in places]
    d = torch.full((9, H, W), -7.0, device="cuda")
    ctx.stitch_device(mode, W, H, places, d[0].data_ptr(), d[1].data_ptr(), ramp=4)
    ctx.close()
    want, acc = np.full((9, H, W), -7.0), np.zeros((10, H, W))
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
    got = d.cpu().numpy()
    if mode == 2:
        want = np.where(acc[0] > 0, acc[1:] / np.where(acc[0] > 0, acc[0], 1), -7.0)
        assert np.abs(got - want).max() < 1e-5  # FP32 sums of a few weighted values in [0, 1]
    else:
        assert np.array_equal(got, want.astype(np.float32))
