// Batched-acceptance search kernel: the reference's search loop
// (QuantizedGraph::search_qg_with_heap, symqglib/qg/qg.hpp:298-344), exact
// for every query, ties included.
//
// One warp per query, persistent over the work queue, as the split kernel:
// the search pool `sp` is the reference's std::priority_queue emulated step
// for step (heap_ops.cuh), and of the result pool `rp` the search keeps only
// what it reads, lowerBound = rp.top().distance, the ef-th smallest accepted
// distance (the largest one while fewer than ef are accepted). The accepted
// nodes at or below the bound are kept sorted in shared memory (the sorted
// pool), and every accepted node is appended, in order, to the query's result
// log in HBM (id, distance, bound after it).
//
// What differs is how one expansion's candidates are decided. The reference
// takes them one by one in list order (qg.hpp:329-335): accept if rp holds
// fewer than ef or lowerBound > distance. Here the warp decides all of them
// at once from one count: candidate j is accepted exactly when fewer than ef
// values of {accepted before this expansion} + {candidates before j in this
// expansion} are <= its distance y_j. (While rp is not full that count is
// below ef. Once it is full, lowerBound is the ef-th smallest accepted value
// L, and y < L is "fewer than ef accepted values <= y"; an earlier candidate
// that was rejected has a value >= the bound of its time >= the bound of any
// later time, so counting it changes no decision, and an earlier accepted one
// counts as it should.) The accepted distances before the expansion that can
// count sit in the sorted pool, so the count is a binary search there plus a
// prefix count over the expansion's candidates. The accepted ones are merged
// into the sorted pool in one step, the bound after each of them is read off
// the merged pool (after the t-th of m accepted it is the value at position
// ef - 1 + m - t once rp is full: the later accepted values are all below
// it), and they enter the search pool in list order.
//
// When the output does not depend on how equal distances sit in rp, the warp
// writes it from the sorted pool; otherwise it replays the log on a result
// heap laid out as libstdc++ leaves it, in its own shared memory (the visited
// cache, candidates, search heap and sorted pool are free by then), checking
// every acceptance against the reference's test and every logged bound
// against rp.top() (replay_result, heap_ops.cuh).
//
// Visited set: a direct-mapped cache of evaluated ids in shared memory (16-bit
// tags, VisitedCache in lqg_kernels.cuh). It may forget an id, never invents one. A forgotten node that is evaluated
// again has its old distance; if it passes the bound now it was accepted
// before and is still in the sorted pool with the same id and distance, and
// it is dropped there.
//
// Lazy mode (ReplayArgs::lazy) keeps no search heap while the smallest
// unpopped distance is unique (the heap's top is then the sorted pool's first
// unpopped entry) and brings it up to date from the logs at a tie (below).
//
// A query whose search pool, sorted pool or log outgrows its capacity goes to
// the exact global-memory kernel through the spill list.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>

#include "heap_ops.cuh"
#include "launch_shape.h"
#include "lqg_internal.h"
#include "lqg_kernels.cuh"
#include "sq8_batch.cuh"
#include "sq8_filter.cuh"

namespace lqg {

// Per-query values that are read once or twice per pop: kept in shared memory,
// so that the search loop's registers hold only what every step needs.
struct WarpState {
    float K, st, E;  // the filter's constants (Sq8Filter)
    uint32_t qi;
    uint32_t pops, calcs;
    float smax, n2;  // the filter's per-index sums
    uint32_t hpush, hpop;  // lazy mode: pushes and pops that the search heap holds
    uint32_t pad[2];
};
static_assert(sizeof(WarpState) == 48, "BatchLayout reserves 48 bytes");

// After a search, a warp's visited cache, candidates, search heap and sorted
// pool (contiguous) can hold a result heap of rcap slots.
__host__ __device__ inline bool batch_replays_in_place(uint32_t deg, uint32_t vbits, uint32_t scap,
                                                       uint32_t acap, uint32_t rcap) {
    return 4 * ((size_t)1 << vbits) + 8 * (size_t)deg + 8 * (size_t)scap + 8 * (size_t)acap >=
           8 * (size_t)rcap;
}

constexpr uint32_t kPopped = 0x80000000u;  // sorted-pool id flag (ids are < 2^31)

// The search heap of a query that runs without one (lazy mode), brought up to
// date: the reference's pushes (every accepted node in order, read from the
// result log) and pops (each after the logged number of pushes) since the heap
// was last up to date (`pushed` pushes and `popped` pops, 0 and 0 at first; sn
// entries). Every replayed pop must return the node that the lazy search popped
// there. Returns the heap's size, or kNoId (heap unusable) when one does not or
// the heap would outgrow its slots. Not inlined: few pops come here, and the
// search loop has to stay in the instruction cache.
static __device__ __noinline__ uint32_t update_search_heap(const heapops::HeapView sp,
                                                           uint32_t sp_max, const uint4* rlog,
                                                           const uint2* plog, uint32_t sn,
                                                           uint32_t pushed, uint32_t popped,
                                                           uint32_t acc_n, uint32_t pops, int lane) {
    using namespace heapops;
    uint32_t i = pushed;
    for (uint32_t j = popped; j <= pops; ++j) {
        const uint2 pj = j < pops ? plog[j] : make_uint2(acc_n, kNoId);
        while (i < pj.x) {
            const uint32_t cnt = min(32u, pj.x - i);
            if (sn + cnt > sp_max) return kNoId;
            const uint4 e = (uint32_t)lane < cnt ? rlog[i + lane] : make_uint4(0, 0, 0, 0);
            for (uint32_t t = 0; t < cnt; ++t) {
                const uint32_t id = __shfl_sync(kFull, e.x, t);
                const uint32_t yb = __shfl_sync(kFull, e.y, t);
                warp_push(sp, sn, make_uint2(id, yb ^ 0x80000000u), lane);  // -distance
            }
            i += cnt;
        }
        if (j < pops) {
            if (sn == 0 || sp.get(0).x != pj.y) return kNoId;
            warp_pop(sp, sn, lane);
        }
    }
    return sn;
}

// replay_result out of the search loop's code, as above. (a and ra are
// __grid_constant__ kernel parameters: nothing is copied.)
static __device__ __noinline__ bool replay_result_call(const SearchArgs& a, const ReplayArgs& ra,
                                                       int64_t qi, uint32_t len,
                                                       const heapops::SharedHeap rp, int lane) {
    return replay_result(a, ra, qi, len, rp, lane);
}

// Number of entries of the sorted values a[0, n) that are <= y, n > 0: a search
// by quarters, without branches or bounds checks (the caller keeps the slots
// past the last entry at +inf, so n is the array's whole length). The three
// loads of a round overlap: 4 rounds of about 65 cycles for 96 slots, where
// halving takes 7 of 69. One search per lane, whatever the number of members; a
// rank by ballots, one member after the other, took 26 instructions per member.
__device__ __forceinline__ uint32_t upper_rank(const float* a, uint32_t n, float y) {
    const float* p = a;
#pragma unroll 1
    while (n > 3) {  // warp-uniform
        const uint32_t q = n >> 2;
        const uint32_t c = (p[q - 1] <= y ? 1u : 0u) + (p[2 * q - 1] <= y ? 1u : 0u) +
                           (p[3 * q - 1] <= y ? 1u : 0u);
        p += c * q;
        n -= 3 * q;  // of the last quarter, the longest
    }
    const uint32_t c = (p[0] <= y ? 1u : 0u) + (n > 1 && p[1] <= y ? 1u : 0u) +
                       (n > 2 && p[2] <= y ? 1u : 0u);
    return (uint32_t)(p - a) + c;
}

// Named barriers of the latency form (barrier 0 is __syncthreads).
__device__ __forceinline__ void named_bar(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// What the warps of the latency form tell each other at the end of a step.
struct PairMerge {    // from the merging warp
    float nd;         // the first unpopped pool entry (+inf: none)
    uint32_t nid;
    float lower;
    uint32_t flags;
    uint32_t next;    // kPairRedo: the node to expand
};
struct PairExpand {   // from an expanding warp
    uint32_t ncand;   // its candidates: ncand from place `start` of the buffer
    uint32_t start;
    uint32_t mb, mid; // its nearest candidate: distance bits, id
    uint32_t single;  // no other candidate at that distance
};
static_assert(sizeof(uint32_t) + 2 * sizeof(PairMerge) + 2 * 3 * sizeof(PairExpand) +
                      sizeof(uint32_t) + 8 <= kLatencyStatic,
              "the messages of three expanding warps, the query and the list length");
constexpr uint32_t kPairFull = 1u;  // rp is full
constexpr uint32_t kPairTie = 2u;   // another unpopped entry at distance nd
constexpr uint32_t kPairHeap = 4u;  // the search heap decides every pop
constexpr uint32_t kPairDone = 8u;  // the query is over
constexpr uint32_t kPairRedo = 16u; // the step's expansion does not count; expand `next`

// NE = 0: one warp per query, blocks of up to 5 query warps. NE > 0: one query
// per block of one merging and NE expanding warps, which work on successive pops
// at the same time (the latency form for batches whose queries all fit on the
// GPU at once).
//
// The latency form. The next pop is known as soon as a pop's candidates have their
// distances: it is the nearest of them if that passes the bound and lies below
// the first unpopped pool entry, else that entry. So while warp 0 merges the
// candidates of one pop, the others already expand the next (list and visited
// cache by warp 1, then bound and exact distances over all of them, a segment of
// the candidates each), with the bound from before the merge (it only falls, and
// the merge tests every candidate again). One barrier per pop, and one more among
// three expanding warps; candidates and messages are double-buffered. Where the next pop is not certain - equal
// smallest distances, or the search heap in use - the expanders wait a step for
// warp 0 to pop. The nearest candidate can be a node that the visited cache forgot and
// that was popped before. A table of the popped ids keeps most of them from being
// expanded again (without it a third of the pops at ef 200 and degree 96 were);
// for the rest, warp 0 finds another first entry after the merge, the expansion is
// discarded (kPairRedo), and its marks in the visited cache are true ones, since
// every neighbour of a popped node has been visited.
//
// WIDE: rows of kWideDim code bytes or more.
//
// What bounds it: instruction issue along one query's dependent steps. A pop
// costs about 1,000 warp instructions and a lone warp issues one every 2.5
// cycles, so the code is written for few instructions, short dependent chains
// and a small instruction footprint (loops over rows and members are not
// unrolled: unrolled, instruction-cache misses took 20 % of the time).
// Registers: 96 let 20 warps live on an SM without spills for rows below 256
// bytes (but for 3 to 17 words at degree 32 to 128); 24 warps at 80 registers and
// fewer are slower (spills). Wider rows and the latency form are bound to fewer
// warps by shared memory, and take 128.
// Device calls, before and after the distance bound, the list prefetch, the
// checked-distinct lists, the 16-bit visited tags, the shorter heap steps and the
// latency form's steps (one B200, us):
//   1M x 128 deg 32 ef 64, 10,000 queries      2,932 -> 2,153
//   200k x 96 deg 32 ef 100, 37 queries          577 ->   347
//   100k x 768 deg 64 ef 128, 2,000 queries    4,750 -> 2,890
//   100k x 960 deg 64 ef 32-512, 2,048        19,750 -> 6,370
//   100k x 100 deg 96 ef 200, 1,777 queries    2,655 -> 1,825
template <int DEGW, bool WIDE, int NE>
__global__ void __maxnreg__(WIDE || NE ? kWideRegs : kNarrowRegs)
    batch_search_kernel(const __grid_constant__ SearchArgs a, const __grid_constant__ ReplayArgs ra) {
    using namespace heapops;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int hw = (int)(threadIdx.x >> 5);
    const bool expander = NE > 0 && hw > 0;
    constexpr uint32_t kThreads = 32u * (1 + NE);  // NE > 0: of a block
    const uint32_t dim = a.dim;
    const uint32_t dpad = (dim + 15u) & ~15u;
    float* pmin = reinterpret_cast<float*>(smem);
    float* pscale = pmin + dpad;
    const uint32_t vbits = a.vbits;
    const uint32_t acap = ra.acap;
    const BatchLayout L = batch_layout(dim, 32 * DEGW, vbits, ra.scap, acap, NE > 0);
    unsigned char* wb = smem + 8u * dpad + (NE ? 0u : hw * L.total);
    float* qs = reinterpret_cast<float*>(wb);
    int8_t* planes = reinterpret_cast<int8_t*>(wb + L.planes);
    volatile WarpState* ws = reinterpret_cast<WarpState*>(wb + L.state);
    const VisitedCache vis{reinterpret_cast<uint16_t*>(wb + L.vis), vbits};
    // candidates: ids, then distances (NE: buffer b starts at 64 DEGW b)
    uint32_t* const cand = reinterpret_cast<uint32_t*>(wb + L.cand);
    float* ad = reinterpret_cast<float*>(wb + L.pool);    // sorted pool: distances
    uint32_t* ai = reinterpret_cast<uint32_t*>(ad + acap);  // and ids
    const uint32_t gw = blockIdx.x * (NE ? 1u : (blockDim.x >> 5)) + (NE ? 0u : hw);
    const HeapView sp{reinterpret_cast<uint2*>(wb + L.heap), ra.sp_global + (size_t)gw * ra.gcap,
                      ra.scap};

    if (a.nlist && *a.nlist == 0) return;  // the batch went to the other form
    for (uint32_t i = threadIdx.x; i < dpad; i += blockDim.x) {
        pmin[i] = i < dim ? a.params[2 * i] : 0.f;
        pscale[i] = i < dim ? a.params[2 * i + 1] : 0.f;
    }
    __syncthreads();

    const float INF = CUDART_INF_F;
    constexpr int NS = NE ? NE : 1;              // segments of an expansion's candidates
    __shared__ uint32_t s_query;                 // NE: the block's query
    __shared__ volatile PairMerge s_pm[2];       // NE: messages of even and odd steps
    __shared__ volatile PairExpand s_pe[2][NS];
    __shared__ volatile uint32_t s_list;         // NE > 1: candidates of the list being expanded
    {
        float smax, n2;
        filter_index_sums(pmin, pscale, dim, lane, smax, n2);
        if (lane == 0 && (NE == 0 || hw == 1)) {
            ws->smax = smax;
            ws->n2 = n2;
        }
        __syncwarp();
    }

    // a query's state (NE: the merging warp's)
    uint32_t qi = 0, ef = 1;
    bool fail = false;
    uint32_t acc_n = 0;  // accepted so far (rp.size() = min(acc_n, ef))
    uint32_t alen = 0;   // sorted-pool entries
    float lower = INF;
    // Lazy mode: no search heap except for pops that meet a tie. The heap's live
    // entries (distance <= lowerBound; the others are never popped) are exactly
    // the unpopped entries of the sorted pool, so while the smallest of them is
    // unique it is the heap's top. `cur` is the first unpopped entry; pops are
    // logged (pushes are the result log) so the heap can be brought up to date
    // when the smallest distance is shared. sn: the heap's size; heap: not lazy.
    bool heap = false;
    uint32_t sn = 0, cur = 0;
    uint32_t pops = 0;     // NE: pops and the query's logs (else in ws, to save registers)
    uint4* rlg = nullptr;
    uint2* plg = nullptr;
    uint32_t pre = kNoId;  // the node whose list v (and sums sv) hold, or that is prefetched
    uint32_t v[DEGW];
    float sv[DEGW];
    auto load_list = [&](uint32_t node) {
        const size_t o = (size_t)node * (32 * DEGW) + lane;
#pragma unroll
        for (int w = 0; w < DEGW; ++w) v[w] = __ldg(a.nbrs + o + 32 * w);
        if (a.esum)
#pragma unroll
            for (int w = 0; w < DEGW; ++w) sv[w] = __ldg(a.esum + o + 32 * w);
    };
    // NE: the popped ids, by linear probing over 8 slots (it may miss one)
    uint32_t* const popped = reinterpret_cast<uint32_t*>(wb + L.popped);
    auto find_popped = [&](uint32_t id, bool insert) -> bool {
        const uint32_t h = (id * 0x9E3779B1u) >> (32 - kPoppedBits);
        for (uint32_t i = 0; i < 8; ++i) {
            uint32_t* const e = popped + ((h + i) & (kPoppedSlots - 1));
            const uint32_t was = *e;
            if (was == id) return true;
            if (was == kNoId) {
                if (insert) *e = id;
                return false;
            }
        }
        return false;
    };
    auto prefetch_list = [&](uint32_t node) {
        if (lane < 2 * DEGW) {
            const size_t o = (size_t)node * (32 * DEGW) + 32 * (lane >> 1);
            if (!(lane & 1))
                prefetch_l1(a.nbrs + o);
            else if (a.esum)
                prefetch_l1(a.esum + o);
        }
    };
    // qg.hpp:329-335 for ncand candidates, in list order
    auto merge = [&](const uint32_t* cid, const float* cd, uint32_t ncand) {
        // qg.hpp:329-335: 32 candidates of the list at a time, in order
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < ncand; c0 += 32) {
            const uint32_t c = c0 + lane;
            const bool valid = c < ncand;
            float y = valid ? cd[c] : INF;
            const uint32_t id = valid ? cid[c] : kNoId;
            // a distance that is not finite goes to the exact kernel; once
            // rp is full it just fails the test, as in the reference
            if (acc_n < ef && __any_sync(kFull, valid && !(y < INF))) {
                fail = true;
                break;
            }
            // members: candidates that can pass (all while rp is not full)
            bool mem = valid && (acc_n < ef || y < lower);
            // The next pop is the nearest member if it lies below the first
            // unpopped entry, else that entry (a tie may decide otherwise):
            // its list goes into L1 during the merge.
            if (NE == 0) {
                const float nd = cur < alen ? ad[cur] : INF;
                pre = cur < alen ? ai[cur] : kNoId;
                const uint32_t yb = mem ? __float_as_uint(y) : 0x7F800000u;
                const uint32_t mb = __reduce_min_sync(kFull, yb);
                if (mb == 0x7F800000u) continue;  // no member
                if (mb < __float_as_uint(nd))
                    pre = __shfl_sync(kFull, id, __ffs(__ballot_sync(kFull, yb == mb)) - 1);
                prefetch_list(pre);
            }
            const float NaN = __uint_as_float(0x7FC00000u);
            if (!mem) y = NaN;  // compares false everywhere
            uint32_t ub = upper_rank(ad, acap, y);
            // a node the visited cache forgot: still pooled, same distance
#pragma unroll 1
            for (uint32_t x = ub; x > 0 && ad[x - 1] == y; --x)
                if ((ai[x - 1] & ~kPopped) == id) {
                    mem = false;
                    y = NaN;
                }
            const unsigned mmask = __ballot_sync(kFull, mem);
            if (mmask == 0) continue;
            // among the members: pc the earlier ones at or below y, before
            // the ones placed ahead (equal ones in list order)
            uint32_t pc = 0, before = 0;
            const int last = 31 - __clz(mmask);
#pragma unroll 2
            for (int s = 0; s <= last; ++s) {
                const float ys = __shfl_sync(kFull, y, s);
                const bool lo = ys < y, le = ys <= y, early = s < lane;
                before += lo || (le && early) ? 1u : 0u;
                pc += le && early ? 1u : 0u;
            }
            const bool acc = mem && ub + pc < ef;
            const unsigned am = __ballot_sync(kFull, acc);
            const uint32_t m = __popc(am);
            if (m == 0) continue;
            if (alen + m > acap || acc_n + m > ra.rlog_cap || (heap && sn + m > ra.scap + ra.gcap)) {
                fail = true;
                break;
            }
            if (am != mmask) {  // rare: only the accepted ones count
                if (!acc) y = NaN;
                before = 0;
#pragma unroll 1
                for (unsigned bm = am; bm; bm &= bm - 1) {
                    const int s = __ffs(bm) - 1;
                    const float ys = __shfl_sync(kFull, y, s);
                    before += ys < y || (ys == y && s < lane) ? 1u : 0u;
                }
            }
            // merge: accepted j goes after the pooled values <= y_j and the
            // accepted ones ahead of it. Rows of 32 slots from the top: the
            // slots taken by accepted ones as a bit mask; every other slot
            // gets the old entry as many places down as accepted ones lie
            // below it.
            const uint32_t pos = ub + before;
            const uint32_t pmin_new = __reduce_min_sync(kFull, acc ? pos : 0xFFFFFFFFu);
            const float old_max = alen ? ad[alen - 1] : -INF;
            uint32_t below = m;  // accepted ones in rows not yet written
#pragma unroll 1
            for (int rr = (int)((alen + m - 1) >> 5); rr >= (int)(pmin_new >> 5); --rr) {
                const unsigned taken = __reduce_or_sync(
                    kFull, acc && (int)(pos >> 5) == rr ? 1u << (pos & 31u) : 0u);
                below -= __popc(taken);
                const uint32_t x = (uint32_t)rr * 32 + lane;
                const uint32_t sh = below + __popc(taken & ((1u << lane) - 1u));
                const bool mv = sh > 0 && x < alen + m && !((taken >> lane) & 1u);
                float xd = 0.f;
                uint32_t xi = 0;
                if (mv) {
                    xd = ad[x - sh];
                    xi = ai[x - sh];
                }
                __syncwarp();
                if (mv) {
                    ad[x] = xd;
                    ai[x] = xi;
                }
                __syncwarp();
            }
            if (acc) {
                ad[pos] = y;
                ai[pos] = id;
            }
            __syncwarp();
            // the first unpopped entry: the one at `cur` moved up, or an
            // accepted one placed before it
            cur = min(cur + __popc(__ballot_sync(kFull, acc && ub <= cur)), pmin_new);
            alen += m;
            const uint32_t acc_new = acc_n + m;
            const float lf = ad[min(acc_new, ef) - 1];
            // the bound after the t-th accepted (qg.hpp:333-334), logged:
            // read off the merged pool once rp is full, before that the
            // largest value so far
            const uint32_t t = __popc(am & ((1u << lane) - 1u)) + 1;
            float lb = 0.f;
            if (acc_n + 1 < ef) {
                float pmax = acc ? y : -INF;  // inclusive prefix maximum
#pragma unroll 1
                for (int o = 1; o < 32; o <<= 1) {
                    const float v = __shfl_up_sync(kFull, pmax, o);
                    if (lane >= o) pmax = fmaxf(pmax, v);
                }
                lb = fmaxf(old_max, pmax);
            }
            if (acc) {
                if (acc_n + t >= ef) lb = ad[ef - 1 + m - t];
                uint4* const rlog = NE ? rlg : ra.rlog + (size_t)ws->qi * ra.rlog_cap;
                rlog[acc_n + t - 1] =
                    make_uint4(id, __float_as_uint(y), __float_as_uint(lb), 0u);
            }
            // rp trims its largest: beyond position ef only ties with the
            // bound stay in the sorted pool
            if (acc_new > ef) {
                uint32_t keep = ef;
                if (ad[ef] == lf) {  // (slots past the last entry hold +inf)
#pragma unroll 1
                    for (uint32_t x0 = ef; x0 < alen; x0 += 32) {
                        const uint32_t x = x0 + lane;
                        const unsigned em = __ballot_sync(kFull, x < alen && ad[x] == lf);
                        keep += __popc(em);
                        if (em != kFull) break;
                    }
                }
                __syncwarp();
#pragma unroll 1
                for (uint32_t x = keep + lane; x < alen; x += 32) ad[x] = INF;
                alen = keep;
            }
            lower = lf;
            acc_n = acc_new;
            // the search pool takes them in list order (qg.hpp:332)
            unsigned bm = heap ? am : 0u;
            while (bm) {
                const int s = __ffs(bm) - 1;
                bm &= bm - 1;
                const uint32_t sid = __shfl_sync(kFull, id, s);
                const float ys = __shfl_sync(kFull, y, s);
                warp_push(sp, sn, make_uint2(sid, __float_as_uint(-ys)), lane);
            }
            __syncwarp();
        }
    };
    // qg.hpp:313-318: the next node in u; false when the search is over or
    // failed. NE: `tie` tells whether the first unpopped entry after it shares
    // its distance with the one after that.
    auto pop = [&](uint32_t& u, bool& tie) -> bool {
        uint32_t nxt = alen;
        tie = false;
        if (!heap) {
            if (cur >= alen) return false;  // nothing live: top > lowerBound or empty
            u = ai[cur];  // in a tie, another node may be popped
            if (NE == 0) {
                pre = u;
                load_list(pre);
            }
            uint32_t nn = alen;  // the unpopped entry after nxt
#pragma unroll 1
            for (uint32_t x0 = cur + 1; x0 < alen; x0 += 32) {
                const uint32_t x = x0 + lane;
                unsigned um = __ballot_sync(kFull, x < alen && !(ai[x] & kPopped));
                if (um && nxt == alen) {
                    nxt = x0 + __ffs(um) - 1;
                    um &= um - 1;
                    if (NE == 0) break;
                }
                if (um) {
                    nn = x0 + __ffs(um) - 1;
                    break;
                }
            }
            const float dn = ad[min(nxt, acap - 1)];
            if (NE > 0) tie = nn < alen && ad[nn] == dn;
            uint32_t at = cur;  // the popped entry
            if (nxt < alen && dn == ad[cur]) {
                // equal smallest distances: the heap layout decides. The heap
                // is brought up to date and gives this pop.
                const size_t lo = (size_t)ws->qi * ra.rlog_cap;
                const uint32_t np = NE ? pops : ws->pops;
                sn = update_search_heap(sp, ra.scap + ra.gcap, ra.rlog + lo, ra.plog + lo, sn,
                                        NE ? ws->hpush : 0, NE ? ws->hpop : 0, acc_n, np, lane);
                if (sn == kNoId || sn == 0) {
                    fail = true;
                    return false;
                }
                if (NE == 0) {
                    // one warp per query: the heap is kept from here on
                    heap = true;
                } else {
                    // beside expanding warps the pool's order lets them go on
                    u = sp.get(0).x;
                    const float d = ad[cur];
                    __syncwarp();
                    warp_pop(sp, sn, lane);
                    if (lane == 0) {
                        ws->hpush = acc_n;
                        ws->hpop = np + 1;
                    }
                    // it is one of the unpopped entries at the smallest distance
                    bool found = false;
#pragma unroll 1
                    for (uint32_t x0 = cur; x0 < alen && !found; x0 += 32) {
                        const uint32_t x = x0 + lane;
                        const unsigned hit =
                            __ballot_sync(kFull, x < alen && ad[x] == d && ai[x] == u);
                        if (hit) {
                            at = x0 + __ffs(hit) - 1;
                            found = true;
                        } else if (ad[min(x0 + 31, alen - 1)] != d) {
                            break;
                        }
                    }
                    if (!found) {
                        fail = true;
                        return false;
                    }
                }
            }
            if (NE > 0 || !heap) {
                __syncwarp();
                if (lane == 0) {
                    ai[at] = u | kPopped;
                    // (pops < accepted nodes <= rlog_cap)
                    if (NE)
                        plg[pops] = make_uint2(acc_n, u);
                    else
                        ra.plog[(size_t)ws->qi * ra.rlog_cap + ws->pops] = make_uint2(acc_n, u);
                }
                if (at == cur)
                    cur = nxt;
                else if (NE > 0)
                    tie = nxt == at ? nn < alen && ad[nn] == ad[cur] : true;
            }
        }
        if (heap) {
            if (sn == 0) return false;
            const uint2 top = sp.get(0);
            if (-__uint_as_float(top.y) > lower) return false;
            warp_pop(sp, sn, lane);
            u = top.x;
        }
        if (NE)
            ++pops;
        else if (lane == 0)
            ws->pops = ws->pops + 1;
        __syncwarp();
        return true;
    };
    // qg.hpp:320-324 for the node whose list is in v: its unvisited neighbours
    // into cid, their sums into cd. Returns their number.
    auto expand = [&](uint32_t* cid, float* cd) -> uint32_t {
        uint32_t ncand = 0;
        // A list of degree > 32 spans DEGW words. Where the index's lists
        // may repeat an id (SearchArgs::distinct): repeats inside a word
        // are caught by match_any (about 400 cycles); a repeat of an id
        // kept by an earlier word is caught by the cache, unless another
        // id kept in this expansion (in its own word or a later one) took
        // its slot: then (rare) later words also compare against the ids
        // already kept, so no node is a candidate twice (qg.hpp:321). The
        // duplicate check of the acceptance step only sees the pool from
        // before these candidates.
        bool lost = false;
        uint32_t kept = 0;  // words of which this lane's id was kept
        const unsigned lt = (1u << lane) - 1u;
#pragma unroll
        for (int w = 0; w < DEGW; ++w) {
            const uint32_t k = vis.key(v[w]);
            uint16_t* const sl = vis.slot(k);
            const uint16_t tag = vis.tag(k);
            bool keep = *sl != tag;
            if (!a.distinct) {
                const unsigned mm = __match_any_sync(kFull, v[w]);  // all lanes
                keep = keep && (mm & lt) == 0;
                if (DEGW > 1 && w > 0 && lost && keep)
                    for (uint32_t j = 0; j < ncand; ++j)
                        if (cid[j] == v[w]) {
                            keep = false;
                            break;
                        }
            }
            const unsigned kb = __ballot_sync(kFull, keep);
            if (keep) {
                const uint32_t at = ncand + __popc(kb & lt);
                *sl = tag;
                cid[at] = v[w];
                cd[at] = sv[w];
            }
            ncand += __popc(kb);
            __syncwarp();
            if (DEGW > 1 && w + 1 < DEGW && !a.distinct) {
                kept |= keep ? 1u << w : 0u;
                bool gone = false;
#pragma unroll
                for (int e = 0; e <= w; ++e) {
                    const uint32_t ke = vis.key(v[e]);
                    gone |= ((kept >> e) & 1u) && *vis.slot(ke) != vis.tag(ke);
                }
                lost = lost || __any_sync(kFull, gone);
            }
        }
        if (lane == 0) ws->calcs = ws->calcs + ncand;
        return ncand;
    };
    // qg.hpp:325-328: drops (once rp is full) the candidates that certainly fail
    // the bound, and measures the others. Returns their number.
    auto measure = [&](uint32_t* cid, float* cd, uint32_t ncand, bool full, float bound) -> uint32_t {
        if (full && a.esum && ncand > 0) {
            const Sq8Filter f{ws->K, ws->st, ws->E};
            ncand = filter_candidates<WIDE>(a, f, bound, planes, cid, cd, ncand, lane);
        }
        eval_list(a, cid, cd, ncand, qs, pmin, pscale, lane);
        __syncwarp();
        return ncand;
    };

    for (;;) {
        if constexpr (NE > 0) {
            named_bar(1, kThreads);  // the last query's output is written
            if (threadIdx.x == 0) s_query = atomicAdd(a.qhead, 1u);
            named_bar(1, kThreads);
            qi = s_query;
        } else {
            if (lane == 0) qi = atomicAdd(a.qhead, 1u);
            qi = __shfl_sync(kFull, qi, 0);
        }
        if (qi >= (a.nlist ? *a.nlist : (uint32_t)a.m)) break;
        if (a.qlist) qi = (uint32_t)a.qlist[qi];
        ef = min(query_ef(a, qi), ra.efcap);  // efcap <= acap - 32
        if (!expander) {
#pragma unroll 1
            for (uint32_t i = lane; i < acap; i += 32) ad[i] = INF;  // past the last entry: +inf
        }
        if (NE == 0 || hw == 1) {
            const float* q = a.queries + (size_t)qi * dim;
#pragma unroll 1
            for (uint32_t i = lane; i < dpad; i += 32) qs[i] = i < dim ? q[i] : 0.f;
#pragma unroll 1
            for (uint32_t i = 4 * lane; i < (1u << vbits); i += 128)
                *reinterpret_cast<uint4*>(vis.s + 2 * i) = make_uint4(0, 0, 0, 0);
            if (NE)
                for (uint32_t i = 4 * lane; i < kPoppedSlots; i += 128)
                    *reinterpret_cast<uint4*>(popped + i) = make_uint4(kNoId, kNoId, kNoId, kNoId);
            __syncwarp();
            const Sq8Filter f =
                filter_prepare(qs, pmin, pscale, dim, ws->smax, ws->n2, planes, lane);
            if (lane == 0) {
                ws->K = f.K;
                ws->st = f.st;
                ws->E = f.E;
                ws->qi = qi;
                ws->pops = 0;
                ws->calcs = 1;
                ws->hpush = ws->hpop = 0;
                // qg.hpp:305-311: the entry point seeds both pools and is
                // visited; here it is the first round's only candidate
                cand[0] = a.entry;
                const uint32_t k = vis.key(a.entry);
                *vis.slot(k) = vis.tag(k);
            }
            __syncwarp();
            eval_list(a, cand, reinterpret_cast<float*>(cand + 32 * DEGW), 1, qs, pmin, pscale, lane);
        }
        __syncwarp();
        fail = false;
        acc_n = alen = 0;
        lower = INF;
        heap = !ra.lazy;
        sn = cur = 0;
        pre = kNoId;
        pops = 0;
        if (NE) {
            rlg = ra.rlog + (size_t)qi * ra.rlog_cap;
            plg = ra.plog + (size_t)qi * ra.rlog_cap;
        }

        if constexpr (NE == 0) {
            float* const cd = reinterpret_cast<float*>(cand + 32 * DEGW);
            uint32_t ncand = 1;
            for (;;) {
                merge(cand, cd, ncand);
                uint32_t u = kNoId;
                bool tie;
                if (fail || !pop(u, tie)) break;
                if (u != pre || heap) load_list(u);
                ncand = measure(cand, cd, expand(cand, cd), acc_n >= ef, lower);
            }
        } else {
            // step 0: the entry point's distance (warp 1); nothing to merge
            if (lane == 0) {
                if (expander) {
                    volatile PairExpand& e = s_pe[0][hw - 1];
                    e.ncand = hw == 1 ? 1u : 0u;
                    e.start = 0;
                    e.mb = hw == 1 ? cand[32 * DEGW] : 0x7F800000u;
                    e.mid = a.entry;
                    e.single = 1;
                } else {
                    s_pm[0].nd = INF;
                    s_pm[0].nid = ~0u;
                    s_pm[0].lower = INF;
                    s_pm[0].flags = heap ? kPairHeap : 0u;
                    s_pm[0].next = ~0u;
                }
            }
            uint32_t b = 0, seg = 0;
            bool tie = false;
            for (;;) {
                named_bar(1, kThreads);  // the candidates in buffer b, warp 0's message b
                const uint32_t flags = s_pm[b].flags;
                if (flags & kPairDone) break;
                const float bound = s_pm[b].lower;
                // the node to expand in this step (kNoId: warp 0 has to pop first)
                uint32_t x = kNoId;
                if (flags & kPairRedo) {
                    x = s_pm[b].next;
                } else if (!(flags & kPairHeap)) {
                    const uint32_t nd = __float_as_uint(s_pm[b].nd);
                    uint32_t mb = 0x7F800000u, mid = ~0u, single = 0;
#pragma unroll
                    for (int i = 0; i < NS; ++i) {
                        const uint32_t m = s_pe[b][i].mb;
                        if (m == mb) single = 0;
                        if (m < mb) {
                            mb = m;
                            mid = s_pe[b][i].mid;
                            single = s_pe[b][i].single;
                        }
                    }
                    if ((flags & kPairFull) && !(__uint_as_float(mb) < bound)) mb = 0x7F800000u;
                    if (mb < nd)
                        x = single ? mid : ~0u;
                    else if (nd < mb)
                        x = flags & kPairTie ? ~0u : (uint32_t)s_pm[b].nid;
                }
                uint32_t* const cb = cand + 64 * DEGW * b;         // of the last step
                uint32_t* const cn = cand + 64 * DEGW * (b ^ 1u);  // of this one
                if (expander) {
                    uint32_t n = 0, mb = 0x7F800000u, mid = ~0u, same = 0;
                    if (x != kNoId) {
                        float* const cd = reinterpret_cast<float*>(cn + 32 * DEGW);
                        uint32_t total = 0;
                        if (hw == 1) {
                            load_list(x);
                            if (lane == 0) find_popped(x, true);
                            total = expand(cn, cd);
                        }
                        uint32_t s0 = 0;
                        n = total;
                        if (NE > 1) {
                            if (hw == 1 && lane == 0) s_list = total;
                            __syncwarp();
                            named_bar(2, 32 * NE);  // the expanders: list and sums are there
                            total = s_list;
                            const uint32_t w = (total + NE - 1) / NE;
                            s0 = min((hw - 1) * w, total);
                            n = min(w, total - s0);
                        }
                        n = measure(cn + s0, cd + s0, n, flags & kPairFull, bound);
                        for (uint32_t c0 = 0; c0 < n; c0 += 32) {
                            const uint32_t c = c0 + lane;
                            const uint32_t yb = c < n && !find_popped(cn[s0 + c], false)
                                                    ? __float_as_uint(cd[s0 + c])
                                                    : 0xFFFFFFFFu;
                            const uint32_t m = __reduce_min_sync(kFull, yb);
                            const unsigned at = __ballot_sync(kFull, yb == m);
                            if (m == mb) ++same;
                            if (m < mb) {
                                mb = m;
                                mid = cn[s0 + c0 + __ffs(at) - 1];
                                same = __popc(at) > 1;
                            }
                        }
                        if (mid != kNoId) prefetch_list(mid);
                        seg = s0;
                    }
                    if (lane == 0) {
                        volatile PairExpand& e = s_pe[b ^ 1u][hw - 1];
                        e.ncand = n;
                        e.start = seg;
                        e.mb = mb;
                        e.mid = mid;
                        e.single = same == 0;
                    }
                } else {
                    uint32_t nf = 0, u = kNoId;
                    if (!(flags & kPairRedo)) {  // else: nothing to merge, x is popped
                        tie = false;
#pragma unroll 1
                        for (int i = 0; i < NS && !fail; ++i) {
                            const uint32_t s0 = s_pe[b][i].start;
                            merge(cb + s0, reinterpret_cast<float*>(cb + 32 * DEGW) + s0, s_pe[b][i].ncand);
                        }
                        if (fail || !pop(u, tie))
                            nf = kPairDone;
                        else if (u != x)
                            nf = kPairRedo;
                    }
                    if (tie) nf |= kPairTie;  // (kept through a step without a pop)
                    float nd = INF;
                    uint32_t nid = ~0u;
                    if (!heap && cur < alen) {
                        nd = ad[cur];
                        nid = ai[cur];
                        prefetch_list(nid);
                    }
                    if (lane == 0) {
                        s_pm[b ^ 1u].nd = nd;
                        s_pm[b ^ 1u].nid = nid;
                        s_pm[b ^ 1u].lower = lower;
                        s_pm[b ^ 1u].flags =
                            nf | (acc_n >= ef ? kPairFull : 0u) | (heap ? kPairHeap : 0u);
                        s_pm[b ^ 1u].next = u;
                    }
                }
                __syncwarp();
                b ^= 1u;
            }
            if (expander) continue;
        }

        qi = ws->qi;
        // Output (qg.hpp:340-343). rp pops come out in descending distance;
        // only equal distances make the heap layout decide. So when the
        // sorted pool holds exactly rp (no ties beyond the ef-th entry) and
        // the popped entries (the worst k and the one after them, or the
        // whole pool when it is returned) have distinct distances, the output
        // is read off the pool; otherwise the log is replayed.
        const uint32_t P = min(acc_n, ef);
        bool direct = false;
        if (!fail && !ra.replay_all) {
            const uint32_t k = min(a.kq ? a.kq[qi] : a.k0, a.kstride);
            const uint32_t kk = min(k, P);
            const uint32_t lo = a.pool_ids ? 0u : (P > kk ? P - kk - 1 : 0u);
            bool tie = false;
            for (uint32_t x = lo + lane; x + 1 < P; x += 32) tie |= ad[x] == ad[x + 1];
            direct = alen == P && !__any_sync(kFull, tie);
            if (direct) {
                uint32_t* out = a.ids + (size_t)qi * a.kstride;
                for (uint32_t x = lane; x < k - kk; x += 32) out[x] = kNoId;
                for (uint32_t x = P - kk + lane; x < P; x += 32)
                    out[x + k - P] = ai[x] & ~kPopped;
                if (a.pool_ids) {
                    for (uint32_t x = lane; x < a.pstride; x += 32) {
                        a.pool_ids[(size_t)qi * a.pstride + x] = x < P ? ai[x] & ~kPopped : kNoId;
                        a.pool_d[(size_t)qi * a.pstride + x] = x < P ? ad[x] : INF;
                    }
                }
            }
        }
        if (!fail && !direct && !ra.replay_all &&
            batch_replays_in_place(32 * DEGW, vbits, ra.scap, acap, ra.rcap)) {
            __syncwarp();
            const SharedHeap rph(wb + L.vis);
            fail = !replay_result_call(a, ra, qi, acc_n, rph, lane);
            direct = !fail;
        }
        if (lane == 0) {
            ra.rlen[qi] = fail ? kNoId : (direct ? kRlenDone : acc_n);
            if (fail) {
                const uint32_t i = atomicAdd(ra.nspill, 1u);
                ra.spill[i] = (int32_t)qi;
            }
            if (a.stats) {
                *reinterpret_cast<uint4*>(a.stats + 4 * (size_t)qi) =
                    make_uint4(NE ? pops : ws->pops, ws->calcs, 0u, P);
            }
        }
        __syncwarp();
    }
}

template <int DEGW, bool WIDE, int NE>
cudaError_t batch_launch_as(const SearchArgs& a, const ReplayArgs& ra, int warps, int blocks,
                      cudaStream_t st, int* occ) {
    const size_t dpad = (a.dim + 15u) & ~15u;
    const int areas = NE ? 1 : warps;
    const int threads = NE ? 32 * (1 + NE) : warps * 32;
    const size_t smem =
        8 * dpad +
        (size_t)areas * batch_layout(a.dim, 32 * DEGW, a.vbits, ra.scap, ra.acap, NE > 0).total;
    auto k = batch_search_kernel<DEGW, WIDE, NE>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, threads, smem);
    k<<<blocks, threads, smem, st>>>(a, ra);
    return cudaGetLastError();
}

// Expanders of the latency form: where a pop's expansion costs more than its
// merge (long rows, long lists), three warps share it.
template <int DEGW, bool WIDE>
constexpr int batch_expanders() { return WIDE || DEGW > 1 ? 3 : 1; }

template <int DEGW, bool LATENCY = false>
cudaError_t batch_run(const SearchArgs& a, const ReplayArgs& ra, int warps, int blocks,
                      cudaStream_t st, int* occ) {
    constexpr int NW = LATENCY ? batch_expanders<DEGW, true>() : 0;
    constexpr int NN = LATENCY ? batch_expanders<DEGW, false>() : 0;
    return a.dim >= kWideDim ? batch_launch_as<DEGW, true, NW>(a, ra, warps, blocks, st, occ)
                             : batch_launch_as<DEGW, false, NN>(a, ra, warps, blocks, st, occ);
}

}  // namespace lqg
