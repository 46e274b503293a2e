// Batched SQ8 decode + squared L2 of up to 32 candidates per call, shared by
// the heap and replay search kernels. Bit-exact with the reference's
// evaluation (symqglib/qg/qg.hpp:325-328): decode fma(code, scale, min)
// (sq8.hpp:28-32, contracted by -Ofast), then 16 accumulators
// acc[d % 16] = fma(q - dec, q - dec, acc) in increasing d and the AVX-512
// reduction tree (l2.hpp:16-35), then the scalar tail for D % 16.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lqg_kernels.cuh"

namespace lqg {

// Distances of candidates cid[base + p * (32/G) + g], p < NP, into cd[].
// Lane r of group g owns accumulators [r*A, r*A + A) (A = 16/G); all code
// bytes of a round of U chunks, for all NP passes, are requested before any
// arithmetic: 32 code words per lane in flight (U = 32 / (NP * words per
// chunk), at most 8). Passes with no valid candidate are skipped
// (warp-uniform).
template <int G, int NP>
__device__ __forceinline__ void eval_batch(const SearchArgs& a, const uint32_t* cid, float* cd,
                                           uint32_t base, uint32_t ncand,
                                           const float* __restrict__ qs,
                                           const float* __restrict__ pmin,
                                           const float* __restrict__ pscale, int g, int r) {
    constexpr int A = 16 / G;
    constexpr int W = (A + 3) / 4;
    constexpr int CPP = 32 / G;
    constexpr int UU = 32 / (NP * W);
    constexpr int U = UU < 1 ? 1 : (UU > 8 ? 8 : UU);
    constexpr int AP = A >= 2 ? A / 2 : 1;  // accumulator pairs
    const uint32_t dim = a.dim;
    const uint32_t mul = dim & ~15u;
    const unsigned long long C23 = pk(0x4B000000u, 0x4B000000u);

    const uint8_t* rowp[NP];
    bool valid[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const uint32_t c = base + p * CPP + g;
        valid[p] = c < ncand;
        rowp[p] = a.codes + (size_t)(valid[p] ? cid[c] : 0u) * a.cstride + r * A;
    }
    unsigned long long acc2[NP][AP];
    float acc1[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        acc1[p] = 0.f;
#pragma unroll
        for (int t = 0; t < AP; ++t) acc2[p][t] = 0ull;
    }
#pragma unroll 1
    for (uint32_t b0 = 0; b0 < mul; b0 += 16 * U) {
        uint32_t w[NP][U][W];
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t b = b0 + 16 * u;
                if (valid[p] && b < mul) {
                    load_chunk<A>(rowp[p] + b, w[p][u]);
                } else {
#pragma unroll
                    for (int i = 0; i < W; ++i) w[p][u][i] = 0;
                }
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t b = b0 + 16 * u;
            if (b >= mul) break;
            const uint32_t d0 = b + r * A;
            if constexpr (A >= 2) {
                // query, min and scale pairs: 16-byte loads where a lane owns
                // 4 or more dimensions of the chunk (every caller's arrays
                // start on 16 bytes, and d0 is a multiple of A)
                unsigned long long q2[AP], m2[AP], s2[AP];
                if constexpr (AP >= 2) {
#pragma unroll
                    for (int t = 0; t < AP; t += 2) {
                        const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(qs + d0 + 2 * t);
                        const ulonglong2 mm = *reinterpret_cast<const ulonglong2*>(pmin + d0 + 2 * t);
                        const ulonglong2 ss = *reinterpret_cast<const ulonglong2*>(pscale + d0 + 2 * t);
                        q2[t] = qq.x;
                        q2[t + 1] = qq.y;
                        m2[t] = mm.x;
                        m2[t + 1] = mm.y;
                        s2[t] = ss.x;
                        s2[t + 1] = ss.y;
                    }
                } else {
                    q2[0] = *reinterpret_cast<const unsigned long long*>(qs + d0);
                    m2[0] = *reinterpret_cast<const unsigned long long*>(pmin + d0);
                    s2[0] = *reinterpret_cast<const unsigned long long*>(pscale + d0);
                }
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if (base + p * CPP >= ncand) continue;
#pragma unroll
                    for (int t = 0; t < AP; ++t) {
                        const uint32_t wd = w[p][u][(2 * t) / 4];
                        const int s0 = (2 * t) % 4;
                        const uint32_t lo = __byte_perm(wd, 0x4B000000u, 0x7440u + s0);
                        const uint32_t hi = __byte_perm(wd, 0x4B000000u, 0x7440u + s0 + 1);
                        const unsigned long long c2 = sub2(pk(lo, hi), C23);
                        const unsigned long long dec = fma2(c2, s2[t], m2[t]);
                        const unsigned long long df = sub2(q2[t], dec);
                        acc2[p][t] = fma2(df, df, acc2[p][t]);
                    }
                }
            } else {
                const float qv = qs[d0], mv = pmin[d0], sv = pscale[d0];
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if (base + p * CPP >= ncand) continue;
                    const float c = byte_to_float(w[p][u][0], 0);
                    const float dec = __fmaf_rn(c, sv, mv);
                    const float df = __fsub_rn(qv, dec);
                    acc1[p] = __fmaf_rn(df, df, acc1[p]);
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        if (base + p * CPP >= ncand) break;  // warp-uniform
        float acc[A];
        if constexpr (A >= 2) {
#pragma unroll
            for (int t = 0; t < AP; ++t) upk(acc2[p][t], acc[2 * t], acc[2 * t + 1]);
        } else {
            acc[0] = acc1[p];
        }
        // the AVX-512 reduction tree (l2.hpp:16-35): fold 8, 4, 2, 1
#pragma unroll
        for (int h = 8; h >= 1; h >>= 1) {
            if (h >= A) {
#pragma unroll
                for (int t = 0; t < A; ++t) {
                    const float o = __shfl_down_sync(kFull, acc[t], h / A);
                    acc[t] = __fadd_rn(acc[t], o);
                }
            } else {
#pragma unroll
                for (int t = 0; t < A; ++t)
                    if (t < h) acc[t] = __fadd_rn(acc[t], acc[t + h]);
            }
        }
        float res = acc[0];
        const uint32_t c = base + p * CPP + g;
        if (r == 0 && valid[p]) {
            const uint8_t* row = a.codes + (size_t)cid[c] * a.cstride;
            for (uint32_t d = mul; d < dim; ++d) {
                const float cv = (float)row[d];
                const float dec = __fmaf_rn(cv, pscale[d], pmin[d]);
                const float df = __fsub_rn(qs[d], dec);
                res = __fmaf_rn(df, df, res);
            }
            cd[c] = res;
        }
    }
}

// The same distances for few candidates: 8 lanes per candidate (2 dimensions
// of every 16-byte chunk each), candidates cid[base, base + 4 NP) per call; NP
// rows per lane share the query, minimum and scale loads. Groups past the last
// candidate repeat it (no predicates on the loads). A row goes in blocks of 4
// chunks with no branch inside, so that the loads of a block and the
// arithmetic of its chunks overlap.
template <int NP>
__device__ __forceinline__ void eval_few(const SearchArgs& a, const uint32_t* cid, float* cd,
                                         uint32_t base, uint32_t ncand, const float* __restrict__ qs,
                                         const float* __restrict__ pmin,
                                         const float* __restrict__ pscale, int lane) {
    const int g = lane >> 3, r = lane & 7;
    const uint32_t dim = a.dim;
    const uint32_t mul = dim & ~15u;
    const unsigned long long C23 = pk(0x4B000000u, 0x4B000000u);
    const uint8_t* p[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i)
        p[i] = a.codes + (size_t)cid[min(base + 4 * i + g, ncand - 1)] * a.cstride + 2 * r;
    const float* ql = qs + 2 * r;
    const float* ml = pmin + 2 * r;
    const float* sl = pscale + 2 * r;
    unsigned long long acc[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) acc[i] = 0ull;
    auto load = [&](int i, uint32_t d) -> uint32_t {
        return __ldg(reinterpret_cast<const unsigned short*>(p[i] + d));
    };
    // t = q - dec of this lane's 2 dimensions of the chunk at d, for every row
    auto diff = [&](const uint32_t (&w)[NP], uint32_t d, unsigned long long (&t)[NP]) {
        const unsigned long long q = *reinterpret_cast<const unsigned long long*>(ql + d);
        const unsigned long long m = *reinterpret_cast<const unsigned long long*>(ml + d);
        const unsigned long long s = *reinterpret_cast<const unsigned long long*>(sl + d);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const unsigned long long c = sub2(pk(__byte_perm(w[i], 0x4B000000u, 0x7440u),
                                                 __byte_perm(w[i], 0x4B000000u, 0x7441u)), C23);
            t[i] = sub2(q, fma2(c, s, m));
        }
    };
    uint32_t b = 0;
    if (mul >= 64) {
        uint32_t w[4][NP];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int i = 0; i < NP; ++i) w[u][i] = load(i, 16 * u);
#pragma unroll 1
        for (; b + 64 <= mul; b += 64) {
            uint32_t n[4][NP];
            const uint32_t nb = min(b + 64, mul - 64);  // the next block (the last one again)
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < NP; ++i) n[u][i] = load(i, nb + 16 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                unsigned long long t[NP];
                diff(w[u], b + 16 * u, t);
#pragma unroll
                for (int i = 0; i < NP; ++i) acc[i] = fma2(t[i], t[i], acc[i]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < NP; ++i) w[u][i] = n[u][i];
        }
    }
#pragma unroll 1
    for (; b < mul; b += 16) {
        uint32_t w[NP];
        unsigned long long t[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) w[i] = load(i, b);
        diff(w, b, t);
#pragma unroll
        for (int i = 0; i < NP; ++i) acc[i] = fma2(t[i], t[i], acc[i]);
    }
    // the AVX-512 reduction tree (l2.hpp:16-35): fold 8, 4, 2, 1
    float res[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        float x[2];
        upk(acc[i], x[0], x[1]);
#pragma unroll
        for (int h = 4; h >= 1; h >>= 1)
#pragma unroll
            for (int t = 0; t < 2; ++t) x[t] = __fadd_rn(x[t], __shfl_down_sync(kFull, x[t], h));
        res[i] = __fadd_rn(x[0], x[1]);
    }
    if (mul < dim) {  // warp-uniform: the scalar tail, in increasing dimension
        uint32_t w[NP];
        unsigned long long t[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) w[i] = load(i, mul);
        diff(w, mul, t);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            float x[2];
            upk(t[i], x[0], x[1]);
#pragma unroll 1
            for (uint32_t e = 0; mul + e < dim; ++e) {
                const float df = __shfl_sync(kFull, e & 1 ? x[1] : x[0], (lane & ~7) + (e >> 1));
                res[i] = __fmaf_rn(df, df, res[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NP; ++i)
        if (r == 0 && base + 4 * i + g < ncand) cd[base + 4 * i + g] = res[i];
}

// Distances of cid[0, n) into cd by one warp: 8 candidates at a time, a last
// group of up to 4 at half the work.
__device__ __forceinline__ void eval_list(const SearchArgs& a, const uint32_t* cid, float* cd,
                                          uint32_t n, const float* qs, const float* pmin,
                                          const float* pscale, int lane) {
    uint32_t b = 0;
#pragma unroll 1
    for (; b + 4 < n; b += 8) eval_few<2>(a, cid, cd, b, n, qs, pmin, pscale, lane);
    if (b < n) eval_few<1>(a, cid, cd, b, n, qs, pmin, pscale, lane);
}

}  // namespace lqg
