"""Batches with per-query ef around the rule that picks the search kernel's form
on the device (csrc/order.cu): both forms give the oracle's ids."""
import numpy as np
import pytest

from oracle.oracle import IndexArrays, Oracle, sq8_quantize

pytestmark = pytest.mark.gpu


# all at the largest ef (the one-warp form past the blocks), few long ones (the
# latency form), a single long one, and all at ef 1
@pytest.mark.parametrize("kind", ["same", "few", "single", "one"])
@pytest.mark.parametrize("dim,deg,m", [(48, 32, 3001), (48, 32, 20000), (300, 64, 1201)])
def test_uneven_batches(dim, deg, m, kind):
    import torch

    import liteqg_b200

    rng = np.random.default_rng(m)
    n, k = 1500, 20
    x = rng.integers(0, 24, (n, dim)).astype(np.float32)
    q = rng.integers(0, 24, (m, dim)).astype(np.float32)
    ef = np.full(m, 1 if kind == "one" else 64, np.int32)
    if kind in ("few", "single"):
        ef[:] = 8
        ef[rng.choice(m, m // 50 if kind == "few" else 1, replace=False)] = 100
    ks = np.minimum(ef, k).astype(np.int32)
    nb = np.stack([rng.choice(n, deg, replace=False) for _ in range(n)]).astype(np.uint32)
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    dq, de, dk = (torch.from_numpy(v).cuda() for v in (q, ef, ks))
    ids = torch.full((m, k), -7, dtype=torch.int32, device="cuda")
    for _ in range(2):
        ix.search_device(dq.data_ptr(), m, k, ids.data_ptr(), k, ef=int(ef.max()),
                         ef_ptr=de.data_ptr(), k_ptr=dk.data_ptr(),
                         stream=torch.cuda.current_stream().cuda_stream)
    got = ids.cpu().numpy()
    oracle = Oracle(IndexArrays(n, dim, deg, 7, x, nb, codes, params))
    for e in np.unique(ef):
        rows = np.flatnonzero(ef == e)[-60:]
        kk = min(int(e), k)
        want = oracle.search(q[rows], kk, int(e)).compat
        assert np.array_equal(got[rows, :kk].view(np.uint32), want)
