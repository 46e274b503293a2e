"""The work this library is used for, as cases that can be timed.

``listed()`` are fixed cases, ``draw(rng)`` gives more of the same ranges;
``prepare`` makes one case's inputs and resident index, ``run`` is one call as
a program makes it, ``work`` the bytes and operations a call cannot do
without, ``exact`` the floating outputs in 64 bits.

Kinds of case (``"kind"``):
  one       one query per call, host buffers, the set_ef value
  host      a block of queries per call, host buffers
  pool      the same, with the whole result pool (ids and distances)
  device    a block of queries in device memory, one ef for all
  uneven    a block in device memory with per-query ef and k
  fs_one / fs_device   the FastScan/RaBitQ search, one query / device block
  build     index construction from host vectors
  serve     a burst of requests of mixed k and ef through the serving loop

Data are Gaussian mixtures (integer-valued pixels, plain floats or unit-length
rows) or uniform; search cases search a pruned neighbour graph made here with
torch: per node its pruned nearest neighbours, links into nearby clusters and
a few random links, ids in random order.
"""
import math

import numpy as np
import torch

from liteqg_b200.serving import Server
from liteqg_b200.symphonyqg import Index

EFS = (32, 64, 128, 256, 512)  # the uneven batch's per-query ef
KS = (1, 10, 100)


def listed():
    return [
        # A program that answers one query at a time: latency of a single call.
        dict(name="one-1m128", kind="one", n=1_000_000, d=128, deg=32, data="int", m=1, k=10, ef=64),
        # A small request group of a service: fewer queries than the chip holds.
        dict(name="group-200k96", kind="host", n=200_003, d=96, deg=32, data="float", m=37, k=10, ef=100),
        # The standard batched search, queries and results on the device.
        dict(name="batch-1m128", kind="device", n=1_000_000, d=128, deg=32, data="int", m=10_000, k=10, ef=64),
        # High recall, many results, plain host arrays in and out.
        dict(name="batch-500k128-k100", kind="host", n=500_000, d=128, deg=32, data="int", m=10_000, k=100, ef=256),
        # Embedding vectors of unit length, wide lists.
        dict(name="batch-100k768", kind="host", n=100_000, d=768, deg=64, data="unit", m=2_000, k=10, ef=128),
        # Requests of different effort in one batch, very wide rows.
        dict(name="uneven-100k960", kind="uneven", n=100_000, d=960, deg=64, data="float", m=2_048, k=100, ef=512),
        # Ragged dimension (not a multiple of 16) and batch; whole pools for a re-rank.
        dict(name="pool-100k100", kind="pool", n=100_001, d=100, deg=96, data="float", m=1_777, k=50, ef=200),
        # FastScan codes with exact re-rank: throughput and a single call.
        dict(name="fastscan-250k128", kind="fs_device", n=250_000, d=128, deg=32, data="int", m=10_000, k=10, ef=128),
        dict(name="fastscan-one-100k128", kind="fs_one", n=100_000, d=128, deg=32, data="int", m=1, k=10, ef=64),
        # Index construction: many short rows, and fewer embedding rows.
        dict(name="build-100k64", kind="build", n=100_000, d=64, deg=32, data="uniform", m=0, k=0, ef=200),
        dict(name="build-20k768", kind="build", n=20_000, d=768, deg=64, data="unit", m=0, k=0, ef=400),
        # A burst of single requests through the continuous-batching server.
        dict(name="serve-200k96", kind="serve", n=200_000, d=96, deg=32, data="float", m=16_384, k=100, ef=500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("one", "host", "host", "pool", "device", "device", "uneven", "fs_one", "fs_device", "build", "serve"))
    if kind == "build":
        d = _log(rng, 48, 768)
        # rows and pool sizes whose build costs no more than the listed ones
        n = _log(rng, 5_000, min(60_000, 8_000_000 // d))
        return dict(kind=kind, n=n, d=d, deg=rng.choice((32, 64)), data=rng.choice(("uniform", "int", "float", "unit")),
                    m=0, k=0, ef=_log(rng, 64, 256))
    d = _log(rng, 40, 960)
    n = _log(rng, 20_000, min(1_000_000, 60_000_000 // d))
    data = rng.choice(("int", "float", "unit"))
    if kind.startswith("fs"):
        d = _log(rng, 40, 256)
        n = _log(rng, 20_000, min(250_000, 30_000_000 // d))
    deg = rng.choice((32, 32, 64, 96, 128)) if d <= 128 else rng.choice((32, 64))
    ef = _log(rng, 20, 256) if kind != "serve" else 500
    # queries: down to a handful, up to what the listed batches cost
    m = 1 if kind.endswith("one") else _log(rng, 2, min(10_000, max(64, int(8e9 / (ef * deg * d)))))
    if kind == "pool":
        m = min(m, 2_000)
    if kind == "uneven":
        ef, m = 512, _log(rng, 16, max(64, min(4_096, int(6e10 / (512 * deg * d)))))
    if kind == "serve":
        d, deg, n, m = min(d, 128), 32, min(n, 200_000), _log(rng, 500, 16_384)
    k = 100 if kind in ("uneven", "serve") else min(ef, _log(rng, 1, 100))
    return dict(kind=kind, n=n, d=d, deg=deg, data=data, m=m, k=k, ef=ef)


# -- data ---------------------------------------------------------------------

def _clusters(n):
    return max(1, n // 977)


def _mixture(case, n, centres, gen, cluster):
    d, kind = case["d"], case["data"]
    if kind == "uniform":
        return torch.rand((n, d), generator=gen, device="cuda")
    x = torch.randn((n, d), generator=gen, device="cuda")
    if kind == "int":
        return (centres[cluster] + 20.0 * x).clamp_(0, 255).round_()
    x = centres[cluster] + 0.3 * x
    return torch.nn.functional.normalize(x) if kind == "unit" else x


def _points(case, seed):
    """Base rows [n, d], each one's cluster, and queries [m, d], from the seed."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    n, d = case["n"], case["d"]
    c = _clusters(n)
    if case["data"] == "int":
        centres = 255.0 * torch.rand((c, d), generator=gen, device="cuda")
    else:
        centres = torch.randn((c, d), generator=gen, device="cuda")
    cluster = torch.randperm(n, generator=gen, device="cuda") % c
    base = _mixture(case, n, centres, gen, cluster)
    m = max(case["m"], 1)
    qc = torch.randint(0, c, (m,), generator=gen, device="cuda")
    return base, cluster, _mixture(case, m, centres, gen, qc), gen


def _graph(base, cluster, deg, gen):
    """Neighbour ids [n, deg]: in each list the pruned nearest of the node's
    cluster (a neighbour is passed over when a kept one is closer to it than
    the node is, then the nearest left fill up), links into the nearest
    clusters, random links."""
    n, d = base.shape
    c = int(cluster.max()) + 1
    s = -(-n // c)
    order = torch.argsort(cluster, stable=True)
    size = torch.bincount(cluster, minlength=c)  # s or s - 1 each
    start = torch.cumsum(size, 0) - size
    col = torch.arange(s, device="cuda")
    valid = col[None, :] < size[:, None]
    members = order[(start[:, None] + col[None, :]).clamp_(max=n - 1)]
    far = max(4, deg // 8)
    near = deg - 2 * far
    kk = min(near + near // 2, s - 2)
    near = min(near, kk)
    nbrs = torch.empty((n, deg), dtype=torch.int64, device="cuda")
    step = max(1, int(6e7 // (s * s)))
    inf = float("inf")
    for c0 in range(0, c, step):
        mem, ok = members[c0:c0 + step], valid[c0:c0 + step]
        b = mem.shape[0]
        x = base[mem]
        x = x - x[:, :1]
        sq = (x * x).sum(-1)
        dist = sq[:, :, None] + sq[:, None, :] - 2 * torch.bmm(x, x.transpose(1, 2))
        dist.masked_fill_(~ok[:, None, :], inf)
        dist.diagonal(dim1=1, dim2=2).fill_(inf)
        dn, idx = torch.topk(dist, kk, dim=2, largest=False)
        dn, idx = dn.view(b * s, kk), idx.view(b * s, kk)
        cl = torch.arange(b, device="cuda").repeat_interleave(s)[:, None]
        out = torch.zeros((b * s, kk), dtype=torch.bool, device="cuda")
        for i in range(kk):
            keep = ~out[:, i]
            closer = dist[cl, idx[:, i:i + 1], idx] < dn
            closer[:, :i + 1] = False
            out |= closer & keep[:, None]
        pos = torch.arange(kk, device="cuda")
        take = torch.argsort(out * kk + pos, dim=1)[:, :near]
        loc = torch.gather(idx, 1, take)
        ids = torch.gather(mem, 1, loc.view(b, -1)).view(b * s, near)
        rows = ok.reshape(-1)
        nbrs[mem.reshape(-1)[rows], :near] = ids[rows]
    centre = torch.zeros((c, d), device="cuda").index_add_(0, cluster, base) / size[:, None]
    links = deg - near
    if c > 1:
        close = torch.topk(torch.cdist(centre, centre), min(16, c), largest=False).indices
        pick = torch.randint(0, close.shape[1], (n, links), generator=gen, device="cuda")
        to = close[cluster[:, None], pick]
        nbrs[:, near:] = members[to, torch.randint(0, s - 1, (n, links), generator=gen, device="cuda")]
    rnd = max(1, links // 2) if c > 1 else links
    nbrs[:, deg - rnd:] = torch.randint(0, n, (n, rnd), generator=gen, device="cuda")
    # every list holds distinct ids and not its own node: links that repeat are drawn again
    own = torch.arange(n, device="cuda")[:, None]
    while True:
        ids, at = torch.sort(nbrs, dim=1, stable=True)
        again = torch.zeros_like(ids, dtype=torch.bool)
        again[:, 1:] = ids[:, 1:] == ids[:, :-1]
        again = torch.zeros_like(again).scatter_(1, at, again) | (nbrs == own)
        bad = int(again.sum())
        if bad == 0:
            return nbrs
        nbrs[again] = torch.randint(0, n, (bad,), generator=gen, device="cuda")


def _encode(base):
    lo, hi = base.min(0).values, base.max(0).values
    scale = (hi - lo) / 255.0
    safe = torch.where(scale > 0, scale, torch.ones_like(scale))
    codes = ((base - lo) / safe).round_().clamp_(0, 255).to(torch.uint8)
    return codes, torch.stack((lo, scale), 1)


def _index_arrays(case, seed):
    base, cluster, queries, gen = _points(case, seed)
    nbrs = _graph(base, cluster, case["deg"], gen)
    entry = int(torch.argmin(((base - base.mean(0)) ** 2).sum(1)))
    codes, params = _encode(base)
    return base, queries, entry, nbrs, codes, params


# -- the cases ------------------------------------------------------------------

def prepare(case, seed):
    kind, n, d, deg = case["kind"], case["n"], case["d"], case["deg"]
    ix = Index("QG", "L2", n, d, deg)
    if kind == "build":
        return dict(kind=kind, ix=ix, data=_points(case, seed)[0].cpu().numpy(), ef=case["ef"])
    base, queries, entry, nbrs, codes, params = _index_arrays(case, seed)
    fastscan = kind.startswith("fs")
    ix.set_arrays(entry, base.cpu().numpy() if fastscan else None, nbrs.to(torch.int32).cpu().numpy(), codes.cpu().numpy(),
                  params.cpu().numpy())
    if fastscan:
        ix.fastscan_build(seed=1)
    ix.set_ef(case["ef"])
    st = dict(kind=kind, ix=ix, m=case["m"], k=case["k"], ef=case["ef"])
    rng = np.random.RandomState(seed % (1 << 31))
    if kind in ("device", "uneven", "fs_device"):
        st["q"] = queries.contiguous()
        st["ids"] = torch.empty((case["m"], case["k"]), dtype=torch.int32, device="cuda")
        if kind == "uneven":
            st["efs"] = torch.from_numpy(rng.choice(EFS, case["m"]).astype(np.int32)).cuda()
            st["ks"] = torch.from_numpy(rng.choice(KS, case["m"]).astype(np.int32)).cuda()
            # slots past a query's own k are not written: the same in every pass
            st["ids"].fill_(-1)
    else:
        st["q"] = queries.cpu().numpy()
        if kind.endswith("one"):
            st["q"] = st["q"][0]
        if kind == "serve":
            st["efs"] = rng.choice((50, 100, 200, 500), case["m"]).astype(np.uint32)
            st["ks"] = rng.choice((10, 100), case["m"]).astype(np.uint32)
            st["server"] = Server(ix, streams=4, max_k=100, max_ef=512)
    return st


def run(state):
    kind, ix = state["kind"], state["ix"]
    if kind == "build":
        ix.build_index(state["data"], state["ef"], num_iter=3)
        entry, _, nbrs, codes, params = ix.get_arrays()
        return [entry, nbrs, codes, params]
    q, k = state["q"], state["k"]
    if kind in ("one", "host"):
        return ix.search(q, k)
    if kind == "pool":
        ids, (pool_ids, pool_d) = ix.search(q, k, return_pool=True)
        return [ids, pool_ids, pool_d]
    if kind == "fs_one":
        return ix.search_fastscan(q, k)
    if kind == "serve":
        return state["server"].replay(q, state["ks"], state["efs"])[0]
    ids, stream = state["ids"], torch.cuda.current_stream().cuda_stream
    if kind == "fs_device":
        ix.search_fastscan_device(q.data_ptr(), state["m"], k, ids.data_ptr(), k, stream=stream)
    elif kind == "uneven":
        ix.search_device(q.data_ptr(), state["m"], k, ids.data_ptr(), k, ef=state["ef"], ef_ptr=state["efs"].data_ptr(),
                         k_ptr=state["ks"].data_ptr(), stream=stream)
    else:
        ix.search_device(q.data_ptr(), state["m"], k, ids.data_ptr(), k, stream=stream)
    return ids


def _search_work(d, deg, ef, fastscan):
    """Bytes and operations of one search: about ef + 10 expanded nodes and
    two new neighbours in five list slots (fewer in longer lists and larger
    pools, where lists overlap)."""
    pops = ef + 10
    if fastscan:
        p = 1 << (d - 1).bit_length()
        return pops * (4 * d + deg * (p // 8 + 16)) + 4 * d, pops * (3 * d + deg * p // 4)
    evals = 0.4 * pops * deg * min(1.0, 8.0 / math.sqrt(ef)) ** 0.5
    return pops * 4 * deg + evals * d + 4 * d, evals * d * 5


def work(case):
    d, deg, kind = case["d"], case["deg"], case["kind"]
    if kind == "build":
        n = case["n"]
        _, flops = _search_work(d, deg, case["ef"], False)
        pairs = 2 * 96 * 48 * d  # a node's candidates against each other
        return {"bytes": 4 * n * d + 4 * n * deg + n * d, "flops": 3 * n * (flops + 2 * pairs)}
    efs = EFS if kind == "uneven" else (50, 100, 200, 500) if kind == "serve" else (case["ef"],)
    parts = [_search_work(d, deg, e, kind.startswith("fs")) for e in efs]
    m = case["m"] / len(parts)
    out = case["m"] * (4 * case["k"] + (8 * case["ef"] if kind == "pool" else 0))
    return {"bytes": m * sum(b for b, _ in parts) + out, "flops": m * sum(f for _, f in parts)}


def _exact_pool(case, seed):
    """The best-first search's result pool distances in 64 bits: expand the
    nearest unexpanded pool entry, put its unseen neighbours' distances in the
    pool, keep the ef nearest, until every pool entry is expanded."""
    _, queries, entry, nbrs, codes, params = _index_arrays(case, seed)
    m, ef, n = case["m"], case["ef"], case["n"]
    q = queries.double()
    lo, scale = params[:, 0].double(), params[:, 1].double()

    def dist(ids):  # [m, j] -> squared distances to the decoded rows
        return ((codes[ids].double() * scale + lo - q[:, None, :]) ** 2).sum(-1)

    inf = float("inf")
    rows = torch.arange(m, device="cuda")
    seen = torch.zeros((m, n), dtype=torch.bool, device="cuda")
    pool = torch.full((m, ef), inf, dtype=torch.float64, device="cuda")
    ids = torch.zeros((m, ef), dtype=torch.int64, device="cuda")
    todo = torch.zeros((m, ef), dtype=torch.bool, device="cuda")
    ids[:, 0], todo[:, 0] = entry, True
    pool[:, 0] = dist(ids[:, :1])[:, 0]
    seen[:, entry] = True
    while bool(todo.any()):
        at = torch.where(todo, pool, inf).argmin(1)
        live = todo[rows, at]
        todo[rows, at] = False
        nb = torch.sort(nbrs[ids[rows, at]], dim=1).values
        new = ~torch.gather(seen, 1, nb) & live[:, None]
        new[:, 1:] &= nb[:, 1:] != nb[:, :-1]
        seen.scatter_(1, nb, torch.gather(seen, 1, nb) | live[:, None])
        dn = torch.where(new, dist(nb), inf)
        pool, take = torch.sort(torch.cat((pool, dn), 1), dim=1, stable=True)
        pool, take = pool[:, :ef], take[:, :ef]
        ids = torch.gather(torch.cat((ids, nb), 1), 1, take)
        todo = torch.gather(torch.cat((todo, new), 1), 1, take) & (pool < inf)
    return pool


def exact(case, seed):
    if case["kind"] == "pool":
        return [None, None, _exact_pool(case, seed)]
    if case["kind"] == "build":
        x = _points(case, seed)[0].double()
        lo, hi = x.min(0).values, x.max(0).values
        return [None, None, None, torch.stack((lo, (hi - lo) / 255.0), 1)]
    return None  # ids only
