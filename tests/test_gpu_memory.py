"""The sums of the distance bound are a reserve: where device memory ends, work
areas and other indexes get their place, unless a captured graph reads them."""
import contextlib

import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu

MB = 1 << 20
N, DIM, DEG = 400_000, 33, 128  # 205 MB of lists, as much of sums, 19 MB of codes


@pytest.fixture(scope="module")
def arrays():
    rng = np.random.default_rng(2)
    x = rng.integers(0, 256, (N, DIM)).astype(np.float32)
    nb = rng.integers(0, N, (N, DEG), dtype=np.uint32)
    codes, params = sq8_quantize(x, 2)
    return IndexArrays(N, DIM, DEG, 7, x, nb, codes, params)


def _index(a):
    import liteqg_b200

    ix = liteqg_b200.Index("QG", "L2", N, DIM, DEG)
    ix.set_arrays(a.entry, a.vectors, a.nbrs, a.codes, a.params)
    return ix


@contextlib.contextmanager
def _little_left(nbytes):
    """All of the device's memory but about nbytes taken."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del taken
        torch.cuda.empty_cache()


def _queries(m):
    return np.random.default_rng(m).integers(0, 256, (m, DIM)).astype(np.float32)


def test_work_areas_get_the_place_of_the_sums(arrays):
    ix, q = _index(arrays), _queries(5)
    want = Oracle(arrays).search(q, 10, 40).compat
    with _little_left(240 * MB):  # a first call's work areas take 310 MB
        assert np.array_equal(ix.search(q, 10, ef=40), want)
    assert np.array_equal(ix.search(q, 10, ef=40), want)


def test_another_index_gets_the_place_of_the_sums(arrays):
    first, q = _index(arrays), _queries(6)
    want = Oracle(arrays).search(q, 10, 40).compat
    assert np.array_equal(first.search(q, 10, ef=40), want)
    with _little_left(120 * MB):
        second = _index(arrays)
        assert np.array_equal(first.search(q, 10, ef=40), want)
    assert np.array_equal(second.search(q, 10, ef=40), want)


def test_a_captured_graph_keeps_them(arrays):
    import torch

    ix, q = _index(arrays), _queries(7)
    want = Oracle(arrays).search(q, 10, 40).compat
    dq = torch.from_numpy(q).cuda()
    ids = torch.empty((7, 10), dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    call = lambda: ix.search_device(dq.data_ptr(), 7, 10, ids.data_ptr(), 10, ef=40, stream=s.cuda_stream)
    call()
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call()
    with _little_left(120 * MB):
        with pytest.raises(Exception, match="allocation"):
            _index(arrays)
        ids.fill_(-1)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(ids.cpu().numpy().view(np.uint32), want)
    del graph
