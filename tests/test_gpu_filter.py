"""The batch kernels' integer distance bound (csrc/sq8_filter.cuh) must never
drop a candidate that the reference accepts, and the visited cache must keep
every node a candidate once: ids, pools and pops equal the oracle's on data
where the bound is tight, useless or overflows, at dimensions around its
64- and 128-byte slices, and on lists that repeat ids across three and four
32-id words."""
import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu

OFF = 0xFFFFFFFF  # small_batch: never the query-per-block form


def _graph(n, deg, rng):
    nb = np.empty((n, deg), np.uint32)
    for i in range(n):
        nb[i] = rng.choice(n - 1, deg, replace=False)
        nb[i][nb[i] >= i] += 1
    return nb


def _check(x, q, nb, ef, small, vbits=0):
    import liteqg_b200

    n, dim = x.shape
    deg = nb.shape[1]
    codes, params = sq8_quantize(x, 2)
    arr = IndexArrays(n, dim, deg, 7, x, nb, codes, params)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    ix.set_tuning(mode=6, small_batch=small, visited_bits=vbits)
    want = Oracle(arr).search(q, 10, ef)
    ids, (pid, pd), st = ix.search(q, 10, ef=ef, return_pool=True, return_stats=True)
    assert np.array_equal(ids, want.compat)
    assert np.array_equal(pid, want.pool_ids)
    assert np.array_equal(pd, want.pool_d)
    assert np.array_equal(st[:, 0], want.pops)


def _data(kind, n, dim, rng):
    x = rng.random((n, dim)).astype(np.float32)
    if kind == "offset":  # distances far below the values' own rounding
        x += np.float32(3e4)
    elif kind == "mixed_scale":  # a few dimensions dwarf the others
        x *= np.float32(10.0) ** rng.integers(-6, 4, dim).astype(np.float32)
    elif kind == "constant_dims":  # zero scales
        x[:, ::2] = 0.25
    elif kind == "huge":  # products overflow FP32: the bound is infinite
        x *= np.float32(3e17)
    elif kind == "tiny":
        x *= np.float32(1e-20)
    elif kind == "integer":
        x = np.rint(x * 255).astype(np.float32)
    return x


@pytest.mark.parametrize("small", [0, OFF])
@pytest.mark.parametrize("kind,dim", [("uniform", 33), ("uniform", 64), ("uniform", 65),
                                      ("integer", 112), ("uniform", 128), ("integer", 129),
                                      ("uniform", 255), ("uniform", 256), ("integer", 321),
                                      ("uniform", 2048), ("offset", 100), ("mixed_scale", 96),
                                      ("constant_dims", 72), ("huge", 48), ("tiny", 80)])
def test_bound_never_drops_an_accepted_candidate(kind, dim, small):
    rng = np.random.default_rng(dim)
    n = 3000
    x = _data(kind, n, dim, rng)
    q = np.concatenate([x[:20], _data(kind, 44, dim, rng)])
    _check(x, q, _graph(n, 32, rng), 48, small)


@pytest.mark.parametrize("small", [0, OFF])
@pytest.mark.parametrize("deg", [64, 96, 128])
def test_repeated_ids_across_words(deg, small):
    """Ids of the first word again in the later ones, a 256-slot-word cache: a
    kept id's slot is often taken within the expansion, by its own word or a
    later one."""
    rng = np.random.default_rng(deg)
    n, dim = 4000, 48
    x = np.rint(rng.random((n, dim)) * 40).astype(np.float32)
    nb = _graph(n, deg, rng)
    for i in range(n):
        for w in range(1, deg // 32):
            nb[i, 32 * w + rng.choice(32, 11, replace=False)] = nb[i, rng.choice(32, 11, replace=False)]
    _check(x, np.rint(rng.random((100, dim)) * 40).astype(np.float32), nb, 100, small, vbits=8)
