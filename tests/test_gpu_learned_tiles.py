"""The network's loss gradient where the 8 x 16 pixel tiles of its kernels are
partly filled or many: the gradient of a batch of copies of one patch is that
many times the patch's gradient.  Every copy runs the same roundings (fields,
subspace sums, bfloat16 output gradients), so the two differ only by the order
of FP32 sums over at most 1e4 pixels per copy: some units of 2^-24 times
sqrt(1e4), 1e-5 of the terms; 1e-4 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,n", [(33, 17, 5), (8, 48, 3), (57, 16, 2), (100, 100, 3), (7, 130, 4)])
def test_gradient_of_copies(H, W, n):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import learned
    rng = np.random.default_rng(17)
    ctx = gpb.Context()
    ctx.learned_set(learned.init_params(4))
    mpb, deg = np.clip(rng.normal(0.2, 0.2, (H, W)), 0, 1), rng.uniform(5, 81, (H, W))
    v, _ = np.linalg.qr(rng.normal(size=(H * W, 9)))

    def grad(k):
        dev = [torch.from_numpy(np.tile(np.float32(a).ravel(), k)).cuda() for a in (mpb, deg, v)]
        loss, g = ctx.learned_grad_device([(H, W)] * k, *[d.data_ptr() for d in dev])
        return loss, g.astype(np.float64)
    one, many = grad(1), grad(n)
    ctx.close()
    assert abs(many[0] - n * one[0]) < 1e-9 * max(1.0, many[0])
    assert np.linalg.norm(many[1] - n * one[1]) < 1e-4 * np.linalg.norm(many[1])
