"""The search kernel's two forms under one size of batch: captures, chunks and the
device's choice between them."""
import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu


# With a bound on ef of 200 and more, the latency form's blocks have room for a larger
# visited cache than the one-warp form's 2,048 slots. The latter forgets nodes, and
# evaluates again those that overlapping lists name again: a query's evaluation count
# tells which form ran it. On B200 the latency form has 1,184 blocks
# at 48 dimensions and degree 32. More than 8,192 queries at ef 512 go in chunks of
# 8,192, each with a choice of its own.
@pytest.mark.parametrize("m,top,long_ones,forms", [
    (3001, 200, 60, ["latency"]),            # few long queries
    (3001, 200, 1, ["latency"]),
    (3001, 200, 3001, ["warp"]),             # all the same
    (12000, 200, 12000, ["warp"]),
    (20000, 200, 60, ["warp"]),              # past 16 per block: no look at all
    (10192, 512, 40, ["latency", "warp"]),   # the long ones in the first chunk
])
def test_the_form_that_runs(m, top, long_ones, forms):
    import liteqg_b200

    rng = np.random.default_rng(m + long_ones)
    n, dim, deg, k, chunk = 30000, 48, 32, 5, 8192 if top == 512 else m
    x = rng.integers(0, 24, (n, dim)).astype(np.float32)
    q = rng.integers(0, 24, (m, dim)).astype(np.float32)
    ef = np.full(m, 16, np.uint32)
    ef[rng.choice(chunk, long_ones, replace=False)] = top
    ring = (np.arange(n)[:, None] + np.r_[-14:0, 1:15, rng.integers(15, n - 15, 4)]) % n
    ids = rng.permutation(n)
    nb = np.empty((n, deg), np.int64)
    nb[ids] = ids[ring]
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb.astype(np.uint32), codes, params)
    ids, st = ix.search(q, k, ef=ef, return_stats=True)
    ix.set_tuning(small_batch=0xFFFFFFFF)
    warp_ids, warp = ix.search(q, k, ef=ef, return_stats=True)
    ix.set_tuning(small_batch=1 << 20)
    latency_ids, latency = ix.search(q, k, ef=ef, return_stats=True)
    assert np.array_equal(ids, warp_ids) and np.array_equal(ids, latency_ids)
    for c, form in enumerate(forms):
        rows = slice(c * chunk, (c + 1) * chunk)
        want, other = (warp, latency) if form == "warp" else (latency, warp)
        assert np.array_equal(st[rows], want[rows]), form
        assert not np.array_equal(st[rows], other[rows]), form
    oracle = Oracle(IndexArrays(n, dim, deg, 7, x, nb.astype(np.uint32), codes, params))
    for e in np.unique(ef):
        rows = np.concatenate([np.flatnonzero(ef == e)[:40], np.flatnonzero(ef == e)[-40:]])
        assert np.array_equal(ids[rows], oracle.search(q[rows], k, int(e)).compat)


def test_capture_with_ef_after_a_call_without():
    """After one eager call of a size, a call of that size allocates nothing,
    whether or not it has a per-query ef: it can be captured."""
    import torch

    import liteqg_b200

    rng = np.random.default_rng(3)
    n, dim, deg, m, k, top = 1500, 48, 32, 2001, 10, 100
    x = rng.integers(0, 24, (n, dim)).astype(np.float32)
    q = rng.integers(0, 24, (m, dim)).astype(np.float32)
    ef = np.full(m, 16, np.int32)
    ef[rng.choice(m, 30, replace=False)] = top
    nb = np.stack([rng.choice(n, deg, replace=False) for _ in range(n)]).astype(np.uint32)
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    dq, de = torch.from_numpy(q).cuda(), torch.from_numpy(ef).cuda()
    ids = torch.full((m, k), -7, dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    ix.search_device(dq.data_ptr(), m, k, ids.data_ptr(), k, ef=top, stream=s.cuda_stream)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ix.search_device(dq.data_ptr(), m, k, ids.data_ptr(), k, ef=top, ef_ptr=de.data_ptr(),
                         stream=s.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    got = ids.cpu().numpy()
    oracle = Oracle(IndexArrays(n, dim, deg, 7, x, nb, codes, params))
    for e in (16, top):
        rows = np.flatnonzero(ef == e)[:60]
        assert np.array_equal(got[rows].view(np.uint32), oracle.search(q[rows], k, e).compat)
    del graph


@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("mode", [5, 6])
def test_lanes_do_not_matter(mode, lanes):
    """The batch kernel has no use for lanes_per_cand: small and large batches run
    with every value that set_tuning takes."""
    import liteqg_b200

    rng = np.random.default_rng(lanes)
    n, dim, deg, k, ef = 1500, 48, 32, 10, 20
    x = rng.integers(0, 24, (n, dim)).astype(np.float32)
    nb = np.stack([rng.choice(n, deg, replace=False) for _ in range(n)]).astype(np.uint32)
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    ix.set_tuning(mode=mode, lanes_per_cand=lanes)
    oracle = Oracle(IndexArrays(n, dim, deg, 7, x, nb, codes, params))
    for m in (1, 40, 4000):
        q = rng.integers(0, 24, (m, dim)).astype(np.float32)
        assert np.array_equal(ix.search(q, k, ef=ef)[-40:], oracle.search(q[-40:], k, ef).compat)
