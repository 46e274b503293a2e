"""The search kernel's two forms under one size of batch: captures, chunks and the
device's choice between them."""
import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu


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
