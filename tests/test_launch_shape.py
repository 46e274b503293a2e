"""The batch kernel's launch shapes (csrc/launch_shape.h): what the host chooses
fits an SM as the hardware counts it."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SM, BLOCK, OWN, UNIT = 228 * 1024, 227 * 1024, 1024, 128  # shared memory of an SM and of a block

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "launch_shape.h"
using namespace lqg;
int main() {
    char op[16];
    unsigned dim, deg, vb, scap, tv, ts, acap;
    unsigned long long n;
    long long m;
    int w;
    // op, index, tuning fields, shape so far, queries, warps (blocks per SM for "latency")
    while (std::scanf("%15s %u %u %llu %u %u %u %u %u %lld %d", op, &dim, &deg, &n, &tv, &ts, &vb,
                      &scap, &acap, &m, &w) == 11) {
        ShapeIndex x{};
        x.dim = dim, x.deg = deg, x.n = n, x.sms = 148;
        x.t.visited_bits = tv, x.t.heap_scap = ts;
        size_t bytes = 0;
        if (!std::strcmp(op, "latency")) {
            latency_shape(x, w, acap, vb, scap);
            bytes = 8 * ((dim + 15u) & ~15u) + batch_layout(dim, deg, vb, scap, acap, true).total;
        } else if (!std::strcmp(op, "fast")) {
            w = fast_warps(x, w);
            vb = least_seen_bits(x);
            bytes = fast_smem_bytes(dim, deg, tv, vb, w);
        } else {
            if (!std::strcmp(op, "launch")) {  // as run_batch goes about it
                std::printf("%zu ", batch_smem_bytes(dim, deg, tv, ts, 32 * 17, 1));  // set_tuning's
                w = batch_warps(x, acap, w, scap);
                vb = batch_visited_bits(x, scap, acap, m, w);
                scap = batch_heap_slots(x, vb, scap, acap, w);
            }
            if (!std::strcmp(op, "bits")) vb = batch_visited_bits(x, scap, acap, m, w);
            if (!std::strcmp(op, "slots")) scap = batch_heap_slots(x, vb, scap, acap, w);
            bytes = batch_smem_bytes(dim, deg, vb, scap, acap, w);
        }
        std::printf("%u %u %zu\n", vb, scap, bytes);
    }
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    """Runs the rules on rows (op, dim, deg, n, tuned visited bits, tuned slots,
    bits, slots, pool slots, queries, warps): rows of (bits, slots, bytes)."""
    d = tmp_path_factory.mktemp("shape")
    (d / "main.cpp").write_text(PROGRAM)
    exe = str(d / "shape")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "liteqg_b200", "csrc"),
                    str(d / "main.cpp"), "-o", exe], check=True)

    def run(rows):
        text = "\n".join(" ".join(str(v) for v in r) for r in rows) + "\n"
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return np.array([[int(v) for v in line.split()] for line in out.splitlines()])

    return run


def _own(dynamic, static):
    """What a resident block takes of an SM."""
    return -(-(dynamic + static + OWN) // UNIT) * UNIT


@pytest.mark.parametrize("deg", [32, 64, 96, 128])
def test_latency_blocks_fit_with_their_messages(shapes, deg):
    static = 176  # the kernel's own __shared__ variables, three expanding warps
    rows, most = [], []
    for dim in (33, 96, 100, 128, 300, 768, 960, 1536, 2048):
        for acap in (96, 128, 192, 320, 576):
            for scap in (256, 4096, 13000, 16376, 16384):
                # resident blocks at the smallest shape, as the occupancy query counts them
                base = 8 * (-(-dim // 16) * 16)
                base += 4 * (-(-dim // 16) * 16) + 2 * (-(-dim // 128) * 128) + 48 + 4096
                base += 16 * deg + 8 * scap + 8 * acap + 4096
                if base + static > BLOCK:
                    continue
                for nb in range(1, min(8, SM // _own(base, static)) + 1):
                    rows.append(("latency", dim, deg, 100000, 10, scap, 10, scap, acap, 1, nb))
                    most.append(nb)
    got = shapes(rows)
    for row, nb, (_, _, dynamic) in zip(rows, most, got):
        assert dynamic + static <= BLOCK, row
        assert nb * _own(dynamic, static) <= SM, row


def _blocks(dim, warps, dynamic):
    """Resident blocks of the one-warp form: registers per thread as compiled."""
    regs = 128 if dim >= 256 else 96
    return min(SM // _own(dynamic, 0), 65536 // (regs * 32 * warps))


@pytest.mark.parametrize("warps", [1, 2, 3, 4, 5])
def test_more_slots_and_bits_only_where_they_are_free(shapes, warps):
    cases = [(dim, deg, acap) for dim in (33, 96, 128, 255, 256, 300, 384, 400, 512, 768, 960, 2048)
             for deg in (32, 64, 128) for acap in (96, 128, 192, 320, 576)]
    plain, more, chosen, bits = (shapes([(op, dim, deg, 100000, 10, 256, 10, s, acap, m, warps)
                                         for dim, deg, acap in cases])
                                 for op, s, m in (("bytes", 256, 1), ("bytes", 384, 1),
                                                  ("slots", 256, 1), ("bits", 256, 1500)))
    for (dim, deg, acap), p, q, c, b in zip(cases, plain, more, chosen, bits):
        before = _blocks(dim, warps, p[2])
        if before < 1:
            continue
        free = q[2] <= BLOCK and _blocks(dim, warps, q[2]) >= before
        assert (c[1] == 384) == free, (dim, deg, acap)
        resident = [_blocks(dim, warps, p[2] + warps * ((4 << x) - 4096)) * warps * 148
                    for x in (11, 12, 13)]
        fits = [x for x, r in zip((11, 12, 13), resident) if r >= 1500]
        assert b[0] == (max(fits) if fits else 10), (dim, deg, acap)


@pytest.mark.parametrize("n", [100000, 2**24, 2**24 + 1, 2**26 + 1, 2**28, 2**29 + 1, 2**31 - 1])
def test_many_ids_need_more_bits_and_still_fit(shapes, n):
    """Every tuning that set_tuning takes launches, whatever the ids need."""
    rows = [("launch", dim, deg, n, tv, ts, 0, ts, acap, 100000, warps)
            for dim in (33, 128, 960, 2048) for deg in (32, 128) for acap in (96, 320, 576)
            for tv in (8, 10, 13) for ts in (256, 1024, 2500, 4096, 9000, 16384) for warps in (1, 3, 5)]
    for row, (accepted, bits, slots, dynamic) in zip(rows, shapes(rows)):
        if accepted > BLOCK:
            continue
        assert dynamic <= BLOCK and slots >= 256, row
        assert n <= 1 << (bits + 16), row  # slot and tag name one id


@pytest.mark.parametrize("n", [100000, 2**25 + 1, 2**26 + 1, 2**31 - 1])
def test_fast_kernel_fits_with_many_ids(shapes, n):
    rows = [("fast", dim, deg, n, tv, 256, 0, 0, 0, 1, warps)
            for dim in (33, 400, 960, 1000, 2048) for deg in (32, 64) for tv in (8, 10, 13)
            for warps in (1, 8, 16)]
    for row, (bits, _, dynamic) in zip(rows, shapes(rows)):
        assert dynamic <= BLOCK and n <= 1 << (bits + 16), row


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 5, 200])
def test_large_rows_and_heaps(m):
    """The largest rows beside a search heap that nearly fills a block."""
    import liteqg_b200
    from oracle.oracle import IndexArrays, Oracle, sq8_quantize

    rng = np.random.default_rng(m)
    n, dim, deg, k, ef = 600, 2048, 32, 10, 200
    x = rng.integers(0, 24, (n, dim)).astype(np.float32)
    q = rng.integers(0, 24, (m, dim)).astype(np.float32)
    nb = np.stack([rng.choice(n, deg, replace=False) for _ in range(n)]).astype(np.uint32)
    codes, params = sq8_quantize(x, 2)
    ix = liteqg_b200.Index("QG", "L2", n, dim, deg)
    ix.set_arrays(7, x, nb, codes, params)
    ix.set_tuning(heap_scap=16376)
    want = Oracle(IndexArrays(n, dim, deg, 7, x, nb, codes, params)).search(q, k, ef).compat
    if m == 1:
        ix.set_ef(ef)
        assert np.array_equal(ix.search(q[0], k), want[0])
    assert np.array_equal(ix.search(q, k, ef=ef), want)
