// Warp-cooperative libstdc++ binary-heap steps on (id, distance bits) pairs,
// shared by the search kernels that keep heaps. comp(x, y) is x.dist < y.dist
// (symqglib/qg/qg.hpp:289-293); the search pool stores -distance.
//   push: sift-up while comp(parent, value) (GCC bits/stl_heap.h
//         __push_heap).
//   pop:  move the last element out, walk a hole from the root to a leaf
//         along the larger child (the right one unless comp(right, left)),
//         then sift the moved element up from there (__pop_heap /
//         __adjust_heap).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lqg_internal.h"
#include "lqg_kernels.cuh"

namespace lqg {
namespace heapops {

__device__ __forceinline__ bool hless(uint2 x, uint2 y) {
    return __uint_as_float(x.y) < __uint_as_float(y.y);
}

// A heap array wholly in shared memory, by its address there: in a function that
// is not inlined a pointer would make every access a generic one.
struct SharedHeap {
    uint32_t s;
    __device__ __forceinline__ explicit SharedHeap(const void* p)
        : s((uint32_t)__cvta_generic_to_shared(p)) {}
    __device__ __forceinline__ uint2 get(uint32_t i) const {
        uint2 v;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];"
                     : "=r"(v.x), "=r"(v.y)
                     : "r"(s + 8 * i)
                     : "memory");
        return v;
    }
    __device__ __forceinline__ void set(uint32_t i, uint2 v) const {
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(s + 8 * i), "r"(v.x), "r"(v.y)
                     : "memory");
    }
};

// A heap array: slots [0, cap) in shared memory, slots >= cap (the deepest
// levels of a large search pool) in a per-warp global-memory area.
struct HeapView {
    SharedHeap s;
    uint2* g;
    uint32_t cap;
    __device__ __forceinline__ HeapView(uint2* smem, uint2* global, uint32_t slots)
        : s(smem), g(global), cap(slots) {}
    __device__ __forceinline__ uint2 get(uint32_t i) const {
        return i < cap ? s.get(i) : g[i - cap];
    }
    __device__ __forceinline__ void set(uint32_t i, uint2 v) const {
        if (i < cap)
            s.set(i, v);
        else
            g[i - cap] = v;
    }
};

// push_heap of v at slot n, all lanes: lane i takes the i-th ancestor of the new
// slot, ((n + 1) >> i) - 1. The value rises past the ancestors up to the first
// that is not less than it; each lane reads off one ballot whether it is among
// them, so the moves need no further exchange.
template <class H>
__device__ __forceinline__ void push_steps(H h, uint32_t& n, uint2 v, int lane) {
    const uint32_t p1 = n + 1;
    const uint32_t a = p1 >> lane;
    bool less = false;
    uint2 anc = v;
    if (lane > 0 && a > 0) {
        anc = h.get(a - 1);
        less = hless(anc, v);
    }
    const unsigned m = __ballot_sync(kFull, less) | 1u;  // (lane 0: the new slot)
    const unsigned upto = (2u << lane) - 1u;
    if ((m & upto) == upto) {  // v passes this level
        if (lane > 0) h.set((p1 >> (lane - 1)) - 1u, anc);
        if (((m >> lane) >> 1 & 1u) == 0) h.set(a - 1, v);  // and stays here
    }
    __syncwarp();
    ++n;
}

// A heap that so far lies in shared memory takes the steps without the choice of
// memory in each access (a push of 350 cycles takes 257).
template <class H>
__device__ __forceinline__ void warp_push(H h, uint32_t& n, uint2 v, int lane) {
    push_steps(h, n, v, lane);
}
__device__ __forceinline__ void warp_push(HeapView h, uint32_t& n, uint2 v, int lane) {
    if (n < h.cap)
        push_steps(h.s, n, v, lane);
    else
        push_steps(h, n, v, lane);
}

// pop_heap + pop_back. __adjust_heap moves the larger child up into the hole as
// far as a leaf, and __push_heap then lifts the last element v from there past
// the moved values that are less than v. These do not increase along the path,
// so v ends where the first of them is less than it, and the values below that
// slot are back where they were: the walk stops there. It goes five levels per
// round: lane i (< 31) takes the i-th node, in breadth-first order, of the
// five-level subtree under the hole, loads its children and decides which one
// the walk would take (left only if comp(right, left), or alone) and whether
// the walk goes on (v does not stay). Two ballots tell each lane whether it is on
// the path. All loads of a round precede its stores and no path node is read
// after it is written, so the moves are the sequential walk's.
// (A lone warp, 256 entries: 729 cycles, 1,012 with the walk to the leaf and back
// on the ballots' bits; a push 225, it took 378.)
template <class H>
__device__ __forceinline__ void pop_steps(H h, uint32_t& n, int lane) {
    const uint32_t size = n;
    if (size > 1) {
        const uint32_t len = size - 1;
        const uint2 v = h.get(len);
        // breadth-first index i: depth k = floor(log2(i + 1)), offset i + 1 - 2^k;
        // anc: its ancestors' bits, lefts: those it lies to the left of
        const uint32_t i1 = (uint32_t)lane + 1u;
        const uint32_t k = 31u - __clz(i1);
        const uint32_t off = i1 - (1u << k);
        unsigned anc = 0, lefts = 0;
#pragma unroll
        for (int t = 1; t <= 4; ++t) {
            const unsigned bit = (1u << (i1 >> t)) >> 1;  // 0 above the root
            anc |= bit;
            if (((i1 >> (t - 1)) & 1u) == 0) lefts |= bit;
        }
        uint32_t hole = 0;
        while (true) {
            const uint32_t node = ((hole + 1u) << k) - 1u + off;
            const uint32_t c = 2 * node + 1;
            bool go = false, left = true;
            uint2 ch = v;
            if (lane < 31 && c < len) {
                const uint2 l = h.get(c);
                ch = l;
                if (c + 1 < len) {
                    const uint2 r = h.get(c + 1);
                    left = hless(r, l);
                    ch = left ? l : r;
                }
                go = !hless(ch, v);
            }
            const unsigned mg = __ballot_sync(kFull, go);
            const unsigned ml = __ballot_sync(kFull, left);
            const bool move = go && (mg & anc) == anc && (ml & anc) == lefts;
            if (move) h.set(node, ch);
            const unsigned mv = __ballot_sync(kFull, move);
            if (mv == 0) break;
            const int last = 31 - __clz(mv);  // the deepest
            hole = __shfl_sync(kFull, left ? c : c + 1, last);
            if (last < 15) break;  // above the fifth level
        }
        if (lane == 0) h.set(hole, v);
        __syncwarp();
    }
    n = size - 1;
}

template <class H>
__device__ __forceinline__ void warp_pop(H h, uint32_t& n, int lane) {
    pop_steps(h, n, lane);
}
__device__ __forceinline__ void warp_pop(HeapView h, uint32_t& n, int lane) {
    if (n <= h.cap)
        pop_steps(h.s, n, lane);
    else
        pop_steps(h, n, lane);
}

}  // namespace heapops

// The result pool of query qi replayed from its log (qg.hpp:329-343) on the
// heap rp (one warp): the logged accepted nodes in order, each checked
// against the reference's acceptance test on this heap (size < ef or top >
// distance) and the logged bound after it against rp.top(); then the output:
// the first k pops (results[k-1-j] = j-th pop) and, if asked, the whole pool
// in ascending order. The log is read 32 entries per coalesced load. Returns
// false (nothing written) when a check fails.
__device__ __forceinline__ bool replay_result(const SearchArgs& a, const ReplayArgs& ra,
                                              int64_t qi, uint32_t len, const heapops::SharedHeap rp,
                                              int lane) {
    using namespace heapops;
    const uint32_t efq = query_ef(a, qi);
    const uint32_t ef = min(max(efq, 1u), ra.efcap);
    const uint32_t k = min(a.kq ? a.kq[qi] : a.k0, a.kstride);
    const uint4* lg = ra.rlog + (size_t)qi * ra.rlog_cap;
    uint32_t n = 0, top = 0;
    bool ok = len > 0 && len <= ra.rlog_cap;
    for (uint32_t b = 0; ok && b < len; b += 32) {
        const uint4 mine = b + lane < len ? __ldcs(lg + b + lane) : make_uint4(0, 0, 0, 0);
        const uint32_t cnt = min(32u, len - b);
        for (uint32_t j = 0; j < cnt; ++j) {
            const uint32_t id = __shfl_sync(kFull, mine.x, j);
            const uint32_t yb = __shfl_sync(kFull, mine.y, j);
            const uint32_t lb = __shfl_sync(kFull, mine.z, j);
            if (!(n < ef || __uint_as_float(top) > __uint_as_float(yb))) {
                ok = false;
                break;
            }
            warp_push(rp, n, make_uint2(id, yb), lane);
            if (n > ef) warp_pop(rp, n, lane);
            top = rp.get(0).y;
            if (top != lb) {
                ok = false;
                break;
            }
        }
    }
    if (!ok) return false;
    const uint32_t P = n, kk = min(k, P);
    uint32_t* out = a.ids + (size_t)qi * a.kstride;
    for (uint32_t x = lane; x < k - kk; x += 32) out[x] = kNoId;
    if (a.pool_ids)
        for (uint32_t x = P + lane; x < a.pstride; x += 32) {
            a.pool_ids[(size_t)qi * a.pstride + x] = kNoId;
            a.pool_d[(size_t)qi * a.pstride + x] = __int_as_float(0x7f800000);
        }
    const uint32_t ex = a.pool_ids ? P : kk;
    for (uint32_t j = 0; j < ex; ++j) {
        const uint2 t = rp.get(0);
        if (lane == 0) {
            if (j < kk) out[k - 1 - j] = t.x;
            if (a.pool_ids && P - 1 - j < a.pstride) {
                a.pool_ids[(size_t)qi * a.pstride + (P - 1 - j)] = t.x;
                a.pool_d[(size_t)qi * a.pstride + (P - 1 - j)] = __uint_as_float(t.y);
            }
        }
        warp_pop(rp, n, lane);
    }
    return true;
}

}  // namespace lqg
