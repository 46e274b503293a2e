"""The warp's heap steps (csrc/heap_ops.cuh): data full of ties, whose output and
pop order the heap layout decides, equals the oracle's at heap sizes around the
edges of a level, of a five-level round and of the shared-memory slots."""
import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 4, 5, 6])
@pytest.mark.parametrize("scap", [256, 257, 1024])
@pytest.mark.parametrize("ef", [1, 2, 3, 31, 32, 33, 62, 63, 64, 511, 512])
def test_ties_at_the_edges_of_levels(ef, scap, mode):
    import liteqg_b200

    rng = np.random.default_rng(ef)
    n, dim, deg = 2000, 40, 32
    x = rng.integers(0, 16, (n, dim)).astype(np.float32)
    q = rng.integers(0, 16, (24, dim)).astype(np.float32)
    nb = np.stack([rng.choice(n, deg, replace=False) for _ in range(n)]).astype(np.uint32)
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    ix.set_tuning(mode=mode, heap_scap=scap, small_batch=0xFFFFFFFF)
    want = Oracle(IndexArrays(n, dim, deg, 7, x, nb, codes, params)).search(q, min(ef, 100), ef)
    ids, (pid, pd), st = ix.search(q, min(ef, 100), ef=ef, return_pool=True, return_stats=True)
    assert np.array_equal(ids, want.compat)
    assert np.array_equal(pid, want.pool_ids)
    assert np.array_equal(pd, want.pool_d)
    assert np.array_equal(st[:, 0], want.pops)
