"""Calls with host buffers, around the size up to which the ids arrive in one copy
with the batch's control words (16,384 ids): the results of the device calls."""
import numpy as np
import pytest

from oracle.oracle import sq8_quantize

pytestmark = pytest.mark.gpu

N, DIM, DEG = 3000, 48, 32


@pytest.fixture(scope="module")
def index():
    import liteqg_b200

    rng = np.random.default_rng(11)
    x = rng.integers(0, 24, (N, DIM)).astype(np.float32)
    nb = np.stack([rng.choice(N, DEG, replace=False) for _ in range(N)]).astype(np.uint32)
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", N, DIM, DEG)
    ix.set_arrays(7, x, nb, codes, params)
    ix.fastscan_build(seed=1)
    return ix


def _device(ix, q, k, ef, fastscan):
    import torch

    dq = torch.from_numpy(q).cuda()
    ids = torch.full((len(q), k), -7, dtype=torch.int32, device="cuda")
    call = ix.search_fastscan_device if fastscan else ix.search_device
    call(dq.data_ptr(), len(q), k, ids.data_ptr(), k, ef=ef,
         stream=torch.cuda.current_stream().cuda_stream)
    return ids.cpu().numpy().view(np.uint32)


# one copy, its edges, more (4.8 MB of ids), and back
@pytest.mark.parametrize("fastscan", [False, True])
def test_sizes_in_a_row(index, fastscan):
    rng = np.random.default_rng(5)
    for m, k in ((1, 1), (5, 10), (16383, 1), (256, 64), (16385, 1), (257, 64), (60000, 20), (3, 10), (256, 64)):
        q = rng.integers(0, 24, (m, DIM)).astype(np.float32)
        search = index.search_fastscan if fastscan else index.search
        got = np.asarray(search(q, k, ef=64)).reshape(m, k)
        assert np.array_equal(got, _device(index, q, k, 64, fastscan)), (m, k)


def test_pools_statistics_and_pinned_buffers(index):
    """Further outputs beside few and many ids; queries that the caller pinned."""
    import torch

    rng = np.random.default_rng(6)
    for m, k, ef in ((200, 10, 33), (1701, 10, 64), (200, 64, 100)):
        q = rng.integers(0, 24, (m, DIM)).astype(np.float32)
        ids, (pid, pd), st = index.search(q, k, ef=ef, return_pool=True, return_stats=True)
        assert np.array_equal(ids, _device(index, q, k, ef, False))
        assert (np.diff(pd, axis=1) >= 0).all() and (pd < np.inf).all() and (pid < N).all()
        # the ids are the first k pops of the pool's heap: its k largest distances
        x = np.sort(pd, axis=1)[:, ef - k:]
        at = np.take_along_axis(pd, np.argmax(pid[:, None, :] == ids[:, :, None], axis=2), axis=1)
        assert np.array_equal(np.sort(at, axis=1), x)
        assert (st[:, 3] == ef).all() and (st[:, 0] > 0).all()
        pinned = torch.from_numpy(q).pin_memory().numpy()
        assert np.array_equal(index.search(pinned, k, ef=ef), ids)
