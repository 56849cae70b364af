"""gpb_ucm_batch over images of very different sizes: each result equal to the
bit to that of the image alone.  Image counts around the 32 and 1024 at which
a CTA's search for its image takes another round."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,large", [(2, 0), (33, 32), (40, 7), (1030, 513)])
def test_one_large_among_small(n, large):
    import gpb
    rng = np.random.default_rng(n)
    small = [rng.random((8, h, w), dtype=np.float32) for h, w in ((2, 2), (2, 65), (9, 7), (33, 2), (17, 20))]
    batch = [small[i % 5] for i in range(n)]
    batch[large] = rng.random((8, 301, 260), dtype=np.float32)
    ctx = gpb.Context()
    got = [m for m, _ in ctx.ucm_batch(batch, double_size=True)]
    alone = [ctx.ucm(p, double_size=True)[0] for p in small]
    want = ctx.ucm(batch[large], double_size=True)[0]
    ctx.close()
    for i, m in enumerate(got):
        assert np.array_equal(m, want if i == large else alone[i % 5]), i
