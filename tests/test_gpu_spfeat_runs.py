"""Superpixel descriptors around the number of label runs per warp up to which
pixels are added up in groups (7): stripes of 5 and 4 pixels, single pixels,
random labels and one superpixel, some of them unlabelled or out of range.
Bit-exact, as in test_gpu_spfeat.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["stripes5", "stripes4", "pixels", "random", "one"])
def test_descriptors_by_runs(orc, kind):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import synth
    H, W = 67, 96
    img = synth.voronoi_image(H, W, 12, 8.0, synth.SEED_BASE + 73)
    cb = synth.make_codebook(img, synth.SEED_BASE + 73, k=8, n_sample=1024)
    ctx = gpb.Context(cb, eig_mode=gpb.EIG_WARM, keep_intermediates=1)
    ctx.compute_batch([synth.pack_bgr(img)])
    texton = ctx.fetch("texton", 0, (H, W), np.uint8)
    rng = np.random.default_rng(9)
    flat = np.arange(H * W)
    labels = {"stripes5": flat // 5 % 50, "stripes4": flat // 4 % 50, "pixels": flat, "one": 0 * flat,
              "random": rng.integers(-2, 60, H * W)}[kind].astype(np.int32)
    n = {"pixels": H * W, "one": 1}.get(kind, 50)
    labels[rng.integers(0, H * W, 40)] = -1
    labels[rng.integers(0, H * W, 40)] = n
    d_lab = torch.from_numpy(labels).cuda()
    out = torch.full((n, 8 + 32 + 4), -1.0, dtype=torch.float64, device="cuda")
    ctx.superpixel_features(0, d_lab.data_ptr(), n, out.data_ptr(), bin_step=8, with_textons=True)
    ctx.close()
    assert np.array_equal(out.cpu().numpy(), orc.superpixel_features(img, texton, labels.reshape(H, W), n, 8, K=8))
