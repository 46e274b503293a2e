// Shared-memory layouts of the batch kernel and the rules that choose its launch
// shape: plain arithmetic, for the kernels, for the host that launches them and
// for tests without a GPU.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/lqg.h"

#ifdef __CUDACC__
#define LQG_HD __host__ __device__
#else
#define LQG_HD
#endif

namespace lqg {

// Shared memory: the most a block may use (static part included), what an SM
// has, and what each resident block takes besides its own (rounded up).
constexpr size_t kBlockBytes = 227 * 1024;
constexpr size_t kSmBytes = 228 * 1024;
constexpr size_t kBlockOwn = 1024, kBlockUnit = 128;
constexpr uint32_t kSmRegs = 65536;

// Rows of at least this many code bytes ("wide") prefetch along the row; the
// batch kernel's instances for them take more registers.
constexpr uint32_t kWideDim = 256;
constexpr uint32_t kNarrowRegs = 96, kWideRegs = 128;  // per thread (batch_kernel.cuh)

// Bytes of one plane of a query's distance bound (sq8_filter.cuh): whole rounds
// of two 64-byte slices, zero past dim.
LQG_HD inline uint32_t filter_plane(uint32_t dim) { return (dim + 127u) & ~127u; }

// Shared memory of one search warp: byte offsets of its parts.
struct BatchLayout {
    uint32_t planes, state, vis, cand, heap, pool, popped, total;
};
constexpr uint32_t kPoppedBits = 10, kPoppedSlots = 1u << kPoppedBits;
LQG_HD inline BatchLayout batch_layout(uint32_t dim, uint32_t deg, uint32_t vbits, uint32_t scap,
                                       uint32_t acap, bool pair = false) {
    BatchLayout L;
    L.planes = 4u * ((dim + 15u) & ~15u);            // after the query
    L.state = L.planes + 2u * filter_plane(dim);     // WarpState
    L.vis = L.state + 48u;                           // visited cache
    L.cand = L.vis + (4u << vbits);                  // candidate ids, distances (pair: two)
    L.heap = L.cand + (pair ? 16u : 8u) * deg;       // search heap
    L.pool = L.heap + 8u * scap;                     // sorted pool: distances, ids
    L.popped = L.pool + 8u * acap;                   // pair: popped ids
    L.total = L.popped + (pair ? 4u * kPoppedSlots : 0u);
    return L;
}

// Static shared memory of a latency-form block (its messages), at most.
constexpr size_t kLatencyStatic = 192;

// Shared memory of a block of `warps` query warps, and of one of the latency form.
inline size_t batch_smem_bytes(uint32_t dim, uint32_t deg, uint32_t vbits, uint32_t scap,
                               uint32_t acap, int warps) {
    return 8 * (size_t)((dim + 15u) & ~15u) +
           (size_t)warps * batch_layout(dim, deg, vbits, scap, acap).total;
}
inline size_t batch_latency_bytes(uint32_t dim, uint32_t deg, uint32_t vbits, uint32_t scap,
                                  uint32_t acap) {
    return 8 * (size_t)((dim + 15u) & ~15u) + batch_layout(dim, deg, vbits, scap, acap, true).total +
           kLatencyStatic;
}

// What the shape of a launch depends on besides the batch.
struct ShapeIndex {
    uint32_t dim, deg;
    uint64_t n;
    int sms;
    lqg_tuning t;
};

// Resident blocks of `warps` query warps per SM, by shared memory and registers.
inline int64_t batch_blocks(const ShapeIndex& x, uint32_t vbits, uint32_t scap, uint32_t acap,
                            int warps) {
    const size_t smem = batch_smem_bytes(x.dim, x.deg, vbits, scap, acap, warps);
    if (smem > kBlockBytes) return 0;
    const uint32_t regs = x.dim >= kWideDim ? kWideRegs : kNarrowRegs;
    return std::min<int64_t>(kSmBytes / ((smem + kBlockOwn + kBlockUnit - 1) / kBlockUnit * kBlockUnit),
                             kSmRegs / (regs * 32 * (uint32_t)warps));
}

// The tuned search-heap slots, an even number: warps' areas follow each other in
// shared memory, and their queries are read 16 bytes at a time.
inline uint32_t heap_slots(const lqg_tuning& t) { return (t.heap_scap + 1u) & ~1u; }

// The tuned visited-cache bits, or what names the index's ids uniquely
// (VisitedCache) if that is more.
inline uint32_t least_visited_bits(const ShapeIndex& x) {
    uint32_t vb = x.t.visited_bits;
    while (vb < 15 && x.n > (1ull << (vb + 16))) ++vb;
    return vb;
}

// Warps of a batch-kernel block, at most `warps`, so that the block launches at the
// least visited bits. (With ids past 2^29 the cache alone may leave too little for
// the tuned slots of a single warp; the heap then spills to global memory earlier.)
inline int batch_warps(const ShapeIndex& x, uint32_t acap, int warps, uint32_t& scap) {
    const uint32_t vb = least_visited_bits(x);
    auto fits = [&] { return batch_smem_bytes(x.dim, x.deg, vb, scap, acap, warps) <= kBlockBytes; };
    while (warps > 1 && !fits()) --warps;
    while (scap > 256 && !fits()) scap = std::max(256u, scap / 2 & ~1u);
    return warps;
}

// Visited-cache bits of a batch-kernel launch of m queries, `warps` per block.
// A larger cache forgets fewer nodes (at ef 200 and degree 96: 10.5 k
// evaluations per query at 10 bits, 6.5 k at 13, 5.6 k without forgetting), but
// costs resident queries: a batch that fills the GPU runs at the tuned 10 bits
// (1M x 128, 10,000 queries at ef 64: 2.15 ms at 10, 2.37 at 11, 3.30 at 12).
// So a batch whose queries all fit at once takes the largest cache they fit
// with, when the tuning field is at its default; other values are taken as they
// are.
inline uint32_t batch_visited_bits(const ShapeIndex& x, uint32_t scap, uint32_t acap, int64_t m,
                                   int warps) {
    const uint32_t vb = least_visited_bits(x);
    if (vb != 10) return vb;
    for (uint32_t b = 13; b > vb; --b)
        if (batch_blocks(x, b, scap, acap, warps) * warps * x.sms >= m) return b;
    return vb;
}

// Search-heap slots of a batch-kernel launch, `warps` per block: half as many
// again as the default where they cost no resident block (10,000 queries of
// integers, 1M x 128 at ef 64 / 500k x 128 at ef 256, ms: 2.07 / 9.35 at 256
// slots, 2.04 / 9.14 at 384, 2.05 / 9.63 at 512, 2.52 / 10.76 at 1,024: more
// slots leave less L1, then fewer blocks).
inline uint32_t batch_heap_slots(const ShapeIndex& x, uint32_t vbits, uint32_t scap, uint32_t acap,
                                 int warps) {
    if (x.t.heap_scap != 256) return scap;
    const int64_t least = std::max<int64_t>(batch_blocks(x, vbits, 256, acap, warps), 1);
    return batch_blocks(x, vbits, 384, acap, warps) >= least ? 384 : 256;
}

// The same for the latency form with nb blocks per SM, where shared memory is
// plentiful: first room for the search heap of a query that meets a tie (past
// its slots in shared memory a push waits for global memory: one tie cost a
// query of 560 us another 350 at 256 slots), then the largest visited cache, up
// to 14 bits (2^15 slots; clearing them costs about 600 cycles per query).
inline void latency_shape(const ShapeIndex& x, int nb, uint32_t acap, uint32_t& vbits,
                          uint32_t& scap) {
    const size_t share = kSmBytes / nb / kBlockUnit * kBlockUnit;
    const size_t budget = std::min(kBlockBytes, share - kBlockOwn);
    auto fits = [&](uint32_t vb, uint32_t c) {
        return batch_latency_bytes(x.dim, x.deg, vb, c, acap) <= budget;
    };
    if (x.t.heap_scap == 256)
        for (uint32_t c = 2048; c > 256; c /= 2)
            if (fits(vbits, c)) {
                scap = c;
                break;
            }
    if (x.t.visited_bits == 10)
        for (uint32_t b = 14; b > vbits; --b)
            if (fits(b, scap)) {
                vbits = b;
                break;
            }
}

// Shared memory of a warp of the fast kernel: the query, its byte planes, the cache
// of evaluated nodes, the place cache (lists of several words), candidate ids,
// distances and places; and of a block.
LQG_HD inline uint32_t fast_warp_bytes(uint32_t dim, uint32_t deg, uint32_t vbits, uint32_t sbits) {
    return 4u * ((dim + 15u) & ~15u) + 2u * filter_plane(dim) + (4u << sbits) +
           (deg > 32 ? 4u << vbits : 0u) + 12u * deg;
}
inline size_t fast_smem_bytes(uint32_t dim, uint32_t deg, uint32_t vbits, uint32_t sbits, int warps) {
    return 8 * (size_t)((dim + 15u) & ~15u) +
           (size_t)warps * fast_warp_bytes(dim, deg, vbits, sbits);
}

// The fewest bits of its cache of evaluated nodes: 9, or what names the index's ids
// uniquely; and the warps of a block, at most `warps`, that launches with them.
inline uint32_t least_seen_bits(const ShapeIndex& x) {
    uint32_t sb = 9;
    while (sb < 15 && x.n > (1ull << (sb + 16))) ++sb;
    return sb;
}
inline int fast_warps(const ShapeIndex& x, int warps) {
    while (warps > 1 && fast_smem_bytes(x.dim, x.deg, x.t.visited_bits, least_seen_bits(x), warps) >
                            kBlockBytes)
        --warps;
    return warps;
}

}  // namespace lqg
