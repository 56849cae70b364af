"""The network's loss gradient where the 8 x 16 pixel tiles of its kernels are
partly filled or many, against the oracle's backward pass with bfloat16 at the
same places.  Tolerance as in the learned-start tests: the whole gradient
within 5% and at cosine > 0.999 (bfloat16 roundings that land differently)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(33, 17)], [(8, 48), (57, 16)], [(100, 100)]])
def test_gradient_at_tile_edges(shapes):
    torch = pytest.importorskip("torch")
    import gpb
    import learned_oracle as lo
    rng = np.random.default_rng(17)
    p = lo.init_params(4)
    lay, _ = lo.param_layout()
    for _, _, bo, _, co in lay:
        p[bo:bo + co] = rng.normal(0, 0.02, co)
    want_loss, want, ins = 0.0, np.zeros(lo.nparams()), []
    for H, W in shapes:
        mpb, deg = np.clip(rng.normal(0.2, 0.2, (H, W)), 0, 1), rng.uniform(5, 81, (H, W))
        v, _ = np.linalg.qr(rng.normal(size=(H * W, 9)))
        f = lo.features(mpb, deg)
        L, dy = lo.subspace_loss(lo.forward(p, f, bf=True), v.reshape(H, W, 9), grad=True)
        want_loss += L
        want += lo.backward(p, f, dy, bf=True)
        ins.append((mpb, deg, v))
    dev = [torch.from_numpy(np.concatenate([np.float32(a[k]).ravel() for a in ins])).cuda() for k in range(3)]
    ctx = gpb.Context()
    ctx.learned_set(p)
    loss, g = ctx.learned_grad_device(shapes, *[d.data_ptr() for d in dev])
    ctx.close()
    g = g.astype(np.float64)
    assert abs(loss - want_loss) < 1e-3 * max(1.0, want_loss)
    assert np.linalg.norm(g - want) / np.linalg.norm(want) < 5e-2
    assert g @ want / (np.linalg.norm(g) * np.linalg.norm(want)) > 0.999
