"""The network's kernels where a CTA takes several tiles (more 8 x 16 tiles than
CTAs in every layer: 120 patches with 3000, 1080 and 480 tiles at the first
three levels).

Forward: weights of -1, 0 and 1 and inputs in eighths, so that every sum spans
at most 15 bits and is exact in FP32 in any order; bfloat16 roundings are then
the oracle's and the fields equal to the bit.

Gradient: a batch of distinct patches of one size against the sum over the
patches alone, whose layers have at most 25 tiles, so no CTA takes a second one.
The roundings of each patch are the same in both (fields, subspace sums, output
gradients); the FP32 sums run in other orders: a few units of 2^-24 times the
square root of 3e5 pixels, 1e-4 of the patches' norms together."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(35, 67), (33, 65), (41, 70), (34, 81)]


def _cuda(torch, arrs):
    return torch.from_numpy(np.concatenate([np.ascontiguousarray(a, np.float32).ravel() for a in arrs])).cuda()


def test_forward_exact_on_many_tiles():
    torch = pytest.importorskip("torch")
    import gpb
    import learned_oracle as lo
    rng = np.random.default_rng(11)
    layout, n = lo.param_layout()
    p = np.zeros(n, np.float32)
    for name, wo, bo, ci, co in layout:
        w = np.zeros((co, 9, ci), np.float32)
        for o in range(co):
            for s in (1, 1, -1):
                w[o, rng.integers(9), rng.integers(2 if name == "e0a" else ci)] = s
        p[wo:bo], p[bo:bo + co] = w.ravel(), rng.integers(0, 3, co) / 4
    shapes = [SIZES[i % 4] for i in range(120)]
    mpb = [rng.integers(0, 9, s) / 8 for s in shapes]
    deg = [81 * rng.integers(0, 9, s) / 8 for s in shapes]
    y = torch.empty((sum(h * w for h, w in shapes), 32), device="cuda")
    ctx = gpb.Context()
    ctx.learned_set(p)
    d = _cuda(torch, mpb), _cuda(torch, deg)
    ctx.learned_forward_device(shapes, d[0].data_ptr(), d[1].data_ptr(), y.data_ptr())
    ctx.close()
    got, at = y.cpu().numpy(), 0
    for i, (h, w) in enumerate(shapes):
        want = lo.forward(p, lo.features(mpb[i], deg[i]), bf=True).reshape(-1, 32)
        assert np.array_equal(got[at:at + h * w], want.astype(np.float32)), i
        at += h * w


def test_gradient_of_many_tiles_is_the_patches_sum():
    torch = pytest.importorskip("torch")
    import gpb
    from gpb import learned
    rng = np.random.default_rng(12)
    h, w, n = 35, 67, 120
    mpb = [np.clip(rng.normal(0.2, 0.2, (h, w)), 0, 1) for _ in range(n)]
    deg = [rng.uniform(5, 81, (h, w)) for _ in range(n)]
    v = [np.linalg.qr(rng.normal(size=(h * w, 9)))[0] for _ in range(n)]
    ctx = gpb.Context()
    ctx.learned_set(learned.init_params(4))

    def grad(ix):
        d = [_cuda(torch, [a[i] for i in ix]) for a in (mpb, deg, v)]
        loss, g = ctx.learned_grad_device([(h, w)] * len(ix), *[x.data_ptr() for x in d])
        return loss, g.astype(np.float64)
    alone = [grad([i]) for i in range(n)]
    loss, g = grad(range(n))
    ctx.close()
    assert abs(loss - sum(a[0] for a in alone)) < 1e-9 * loss
    assert np.linalg.norm(g - sum(a[1] for a in alone)) < 1e-4 * sum(np.linalg.norm(a[1]) for a in alone)
