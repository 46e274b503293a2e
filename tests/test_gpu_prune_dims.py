"""The tensor-core prune (64 dimensions per operand buffer, two buffers past
64) builds the FP32 prune's graph at dimensions around its buffer edges, with
candidate counts from few to more than the prune keeps, and on data with
repeated vectors (equal distances, zero distances)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,deg,ef,kind", [
    (33, 32, 16, "uniform"), (63, 32, 64, "uniform"), (64, 32, 200, "uniform"),
    (65, 64, 100, "uniform"), (127, 32, 128, "gauss"), (128, 64, 200, "gauss"),
    (129, 32, 64, "integer"), (192, 96, 256, "gauss"), (200, 128, 300, "integer"),
    (48, 32, 100, "repeated"), (96, 64, 100, "repeated")])
def test_tensor_core_prune_equals_fp32_prune(dim, deg, ef, kind):
    import liteqg_b200

    rng = np.random.default_rng(dim + ef)
    n = 3000
    if kind == "uniform":
        x = rng.random((n, dim), dtype=np.float32)
    elif kind == "gauss":
        x = rng.normal(0, 1, (n, dim)).astype(np.float32)
    elif kind == "integer":
        x = np.rint(rng.random((n, dim)) * 255).astype(np.float32)
    else:
        x = rng.random((n // 4, dim), dtype=np.float32)[rng.integers(0, n // 4, n)]
    graphs = []
    for pk in (0, 1):
        ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
        ix.build_index(x, ef, num_iter=2, random_edges=4, path_take=16, far_budget=4, pair_kernel=pk)
        graphs.append(ix.get_arrays()[2])
    assert np.array_equal(*graphs)
    srt = np.sort(graphs[0], axis=1)
    assert not (srt[:, 1:] == srt[:, :-1]).any()
