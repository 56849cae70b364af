"""The subspace loss's solve on the host (up to 8 patches) and on the device:
the loss of copies of one patch is that many times the patch's loss in both (the
same FP64 operations in the same order on subspace sums that differ by the order
of FP64 atomics: 1e-12), and both refuse a Gram matrix that is not positive
definite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grad(torch, ctx, shape, n, mpb, deg, v):
    d = [torch.from_numpy(np.tile(np.float32(a).ravel(), n)).cuda() for a in (mpb, deg, v)]
    return ctx.learned_grad_device([shape] * n, *[x.data_ptr() for x in d])


@pytest.mark.parametrize("H,W", [(8, 8), (31, 45), (70, 90)])
def test_loss_of_copies_on_both_sides_of_the_line(H, W):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import learned
    rng = np.random.default_rng(H)
    mpb, deg = np.clip(rng.normal(0.2, 0.2, (H, W)), 0, 1), rng.uniform(5, 81, (H, W))
    v = np.linalg.qr(rng.normal(size=(H * W, 9)))[0]
    ctx = gpb.Context()
    ctx.learned_set(learned.init_params(4))
    one = _grad(torch, ctx, (H, W), 1, mpb, deg, v)[0]
    for n in (8, 9, 16):
        assert abs(_grad(torch, ctx, (H, W), n, mpb, deg, v)[0] - n * one) < 1e-12 * n * one
    ctx.close()


@pytest.mark.parametrize("n", [1, 8, 9])
def test_no_solve_of_nan(n):
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import learned
    rng = np.random.default_rng(1)
    mpb, deg, v = np.full((9, 9), 0.2), rng.uniform(5, 81, (9, 9)), np.linalg.qr(rng.normal(size=(81, 9)))[0]
    p = learned.init_params(4)
    bad = p.copy()
    bad[-1] = np.nan  # the head's last bias: a ReLU would drop it
    ctx = gpb.Context()
    ctx.learned_set(bad)
    with pytest.raises(gpb.GpbError):
        _grad(torch, ctx, (9, 9), n, mpb, deg, v)
    ctx.learned_set(p)
    loss, g = _grad(torch, ctx, (9, 9), n, mpb, deg, v)  # the context stays usable
    ctx.close()
    assert np.isfinite(loss) and np.isfinite(g).all()
