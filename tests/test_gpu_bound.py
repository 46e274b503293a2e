"""The distance bound where one dimension outweighs the others: the other weights
are then rounded alike, so that their rounding errors add up."""
import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu


# mode 1 takes the fast kernel of the index builds, 5 and 6 the batch kernel; one
# query per warp and the latency form
@pytest.mark.parametrize("mode,small_batch", [(1, 0), (5, 0xFFFFFFFF), (6, 0xFFFFFFFF), (6, 1 << 20)])
@pytest.mark.parametrize("span", [100.0, 1000.0, -65025.0])
@pytest.mark.parametrize("dim,deg", [(48, 32), (130, 96), (768, 64)])
def test_one_large_dimension(dim, deg, span, mode, small_batch):
    import liteqg_b200

    rng = np.random.default_rng(dim)
    n, m, k = 1500, 150, 10
    x = (rng.integers(0, 4, (n, dim)) + 0.01 * rng.standard_normal((n, dim))).astype(np.float32)
    x[:, 0] = abs(span) * rng.random(n)
    codes, params = sq8_quantize(x, 2)
    if span < 0:  # a scale of either sign is taken
        params = params.copy()
        params[0] = (abs(span), span / 255.0)
    q = x[rng.integers(0, n, m)].copy()
    q[:, 1:] = np.float32(3.0) * rng.random((m, 1), dtype=np.float32)  # one value in all of them
    nb = np.stack([rng.choice(n, deg, replace=False) for _ in range(n)]).astype(np.uint32)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    ix.set_tuning(mode=mode, small_batch=small_batch)
    oracle = Oracle(IndexArrays(n, dim, deg, 7, x, nb, codes, params))
    for ef in (12, 64, 200):
        want = oracle.search(q, k, ef)
        ids, (pid, pd) = ix.search(q, k, ef=ef, return_pool=True)
        assert np.array_equal(ids, want.compat)
        assert np.array_equal(pid, want.pool_ids)
        assert np.array_equal(pd, want.pool_d)
