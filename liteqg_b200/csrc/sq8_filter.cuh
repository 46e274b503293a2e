// Integer bound on the SQ8 distances of an expansion's candidates.
//
// The exact distance of a candidate (sq8_batch.cuh) costs six instructions per
// pair of dimensions, and once the result pool is full most candidates are
// rejected: about 4 of the 20 unseen neighbours of a pop pass the bound at
// ef 64 on 1M x 128. This filter finds the ones that certainly fail, so that
// only the others are evaluated exactly; results do not change.
//
// In real arithmetic, with t = q - min and the code c,
//   y = sum (q - (min + s c))^2 = sum t^2 - sum g c + sum s^2 c^2,  g = 2 s t.
// sum t^2 is per query, sum s^2 c^2 per node (stored per list slot, beside the
// neighbour id: esum), and sum g c is an integer dot product once g is rounded
// to 16 bits: g = st * G + r, G = 256 hi + lo with hi, lo in [-128, 127], so that
// sum g c = st * sum G c + 128 sum r + sum r (c - 128).
// mma.sync m16n8k32 (u8 x s8, exact 32-bit sums) takes 16 candidates by 32
// dimensions against the two byte planes at once; the even columns hold hi,
// the odd ones lo, so every lane of a row's quad ends with both sums. Lane
// (g, c) of a quad reads 16 contiguous bytes of rows g and g + 8, which are
// the K slices of two instructions; the planes are read at the same offsets.
// tcgen05.mma is no fit here: its smallest tile is 64 rows of one operand in
// shared memory shared by a whole block, while every warp walks its own query
// with 16 to 32 gathered rows per step.
//
// Error bound: A = K + S - st * dot differs from y by at most
//   128 sum |r|          the rounding of g: |r| |c - 128|, with -128 sum r in K
//   + 32 u M             every float rounding in K, S, st * dot and their sum,
//                        u = 2^-24, M = K + sum (255 s)^2 + 256 sum |g|
// and the reference's float distance y' (16 accumulators, at most 150
// roundings, decode rounded at u |dec|) obeys
//   y' >= (1 - 2e-5) y - u^2 1e5 N2,  N2 = sum max(|min|, |min + 255 s|)^2.
// So A > lower (1 + 4e-5) + E, with E the sum of the absolute parts, implies
// y' >= lower: the candidate fails the reference's test. Comparisons with a
// NaN or an infinite bound keep the candidate.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "launch_shape.h"
#include "lqg_kernels.cuh"

namespace lqg {

constexpr float kFilterRel = 1.00004f;

struct Sq8Filter {
    float K;   // sum t^2 - 128 sum r
    float st;  // step of G
    float E;   // absolute part of the bound
};

// Per-index sums of the bound: smax = sum (255 s)^2, n2 = N2. All lanes.
__device__ __forceinline__ void filter_index_sums(const float* pmin, const float* pscale,
                                                  uint32_t dim, int lane, float& smax, float& n2) {
    smax = 0.f;
    n2 = 0.f;
#pragma unroll 1
    for (uint32_t d = lane; d < dim; d += 32) {
        const float s = 255.f * pscale[d], m = pmin[d];
        const float x = fmaxf(fabsf(m), fabsf(m + s));
        smax = fmaf(s, s, smax);
        n2 = fmaf(x, x, n2);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        smax += __shfl_xor_sync(kFull, smax, o);
        n2 += __shfl_xor_sync(kFull, n2, o);
    }
}

// The query's planes (shared memory, 16-byte aligned) and constants. All lanes.
__device__ __forceinline__ Sq8Filter filter_prepare(const float* qs, const float* pmin,
                                                    const float* pscale, uint32_t dim, float smax,
                                                    float n2, int8_t* planes, int lane) {
    const uint32_t dp = filter_plane(dim);
    float gm = 0.f;
#pragma unroll 1
    for (uint32_t d = lane; d < dim; d += 32)
        gm = fmaxf(gm, fabsf(2.f * pscale[d] * (qs[d] - pmin[d])));
    gm = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(gm)));
    Sq8Filter f;
    f.st = gm * (1.f / 32512.f);
    const float inv = gm > 0.f ? 32512.f / gm : 0.f;
    double ks = 0.0;
    float R = 0.f, G1 = 0.f;
#pragma unroll 1
    for (uint32_t d = lane; d < dp; d += 32) {
        int hi = 0, lo = 0;
        if (d < dim) {
            const float t = qs[d] - pmin[d];
            const float g = 2.f * pscale[d] * t;
            const int G = min(max(__float2int_rn(g * inv), -32512), 32512);
            lo = ((G + 128) & 255) - 128;
            hi = (G - lo) >> 8;
            const float r = fmaf(-f.st, (float)G, g);
            ks += (double)t * (double)t - 128.0 * (double)r;
            R += fabsf(r);
            G1 += fabsf(g);
        }
        planes[d] = (int8_t)hi;
        planes[dp + d] = (int8_t)lo;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        ks += __shfl_xor_sync(kFull, ks, o);
        R += __shfl_xor_sync(kFull, R, o);
        G1 += __shfl_xor_sync(kFull, G1, o);
    }
    f.K = (float)ks;
    const float M = fabsf(f.K) + 128.5f * R + smax + 256.f * G1;
    f.E = 1.001f * (128.5f * R + 2e-6f * M + 4e-10f * n2 + 1e-30f);
    return f;
}

__device__ __forceinline__ void imma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16 bytes if `in`; otherwise the registers keep what they hold (the caller
// multiplies them by zero). A predicated load, no branch.
__device__ __forceinline__ uint4 load_slice(const uint8_t* p, bool in) {
    uint4 v;
    asm("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n@p ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];\n}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p), "r"((uint32_t)in));
    return v;
}

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Drops from cid[0, ncand), in place and in order, the candidates that
// certainly fail the bound `lower`. cs[i] is candidate i's sum s^2 c^2. 32
// candidates (two 16-row tiles) at a time, two 64-byte slices of every row per
// round: 8 loads of 16 bytes in flight per lane. Rows longer than a round ask
// L1 for the next round's lines (lane l: row l's line) meanwhile. Tile rows
// past the last candidate read the last one again (no predicates, no further
// memory traffic). Returns how many candidates are left. ncand > 0. All lanes;
// ends synchronised.
// TAGGED: `tag` holds a word per candidate that goes with its id.
template <bool WIDE, bool TAGGED = false>
__device__ __forceinline__ uint32_t filter_candidates(const SearchArgs& a, const Sq8Filter f,
                                                      float lower, const int8_t* planes,
                                                      uint32_t* cid, const float* cs,
                                                      uint32_t ncand, int lane,
                                                      uint32_t* tag = nullptr) {
    const int g = lane >> 2, c = lane & 3;
    const uint32_t dp = filter_plane(a.dim);
    const int8_t* pl = planes + (g & 1) * dp + 16 * c;
    const float T = fmaf(lower, kFilterRel, f.E);
    uint32_t out = 0;
#pragma unroll 1
    for (uint32_t b = 0; b < ncand; b += 32) {
        const bool two = b + 16 < ncand;  // warp-uniform
        const uint32_t last = ncand - 1;
        const uint8_t* row[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            row[i] = a.codes + (size_t)cid[min(b + 8 * i + g, last)] * a.cstride + 16 * c;
        const uint8_t* pf =
            WIDE ? a.codes + (size_t)cid[min(b + lane, last)] * a.cstride + 128 : nullptr;
        int acc[2][4] = {};
#pragma unroll 1
        for (uint32_t o = 0; o < dp; o += 128) {
            uint4 w[4][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool in = o + 64 * h + 16 * c < a.cstride;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    w[i][h] = load_slice(row[i] + o + 64 * h, in && (i < 2 || two));
            }
            if (WIDE && o + 128 < a.cstride && b + lane < ncand) prefetch_l1(pf + o);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 q = *reinterpret_cast<const uint4*>(pl + o + 64 * h);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4 x = w[2 * k][h], y = w[2 * k + 1][h];
                    imma_u8s8(acc[k], x.x, y.x, x.y, y.y, q.x, q.y);
                    imma_u8s8(acc[k], x.z, y.z, x.w, y.w, q.z, q.w);
                }
            }
        }
        // lane (g, c) decides candidate b + 8 c + g: rows g (+ 8 for odd c) of
        // tile c / 2, every lane of the quad holding both sums
        const int hi = c & 2 ? (c & 1 ? acc[1][2] : acc[1][0]) : (c & 1 ? acc[0][2] : acc[0][0]);
        const int lo = c & 2 ? (c & 1 ? acc[1][3] : acc[1][1]) : (c & 1 ? acc[0][3] : acc[0][1]);
        const uint32_t x = b + 8 * c + g;
        const float A = fmaf(-f.st, fmaf((float)hi, 256.f, (float)lo), f.K + cs[min(x, last)]);
        const unsigned m = __ballot_sync(kFull, x < ncand && !(A > T));
        // lane l takes candidate b + l in list order: decided by lane 4 (l % 8) + l / 8
        const bool keep = (m >> (4 * (lane & 7) + (lane >> 3))) & 1u;
        const unsigned k = __ballot_sync(kFull, keep);
        const uint32_t id = keep ? cid[b + lane] : 0u;
        const uint32_t tg = TAGGED && keep ? tag[b + lane] : 0u;
        __syncwarp();
        if (keep) {
            const uint32_t at = out + __popc(k & ((1u << lane) - 1u));
            cid[at] = id;
            if (TAGGED) tag[at] = tg;
        }
        out += __popc(k);
        __syncwarp();
    }
    return out;
}

}  // namespace lqg
