// Work order of a batch: the queries expected to run longest first.
//
// The search kernels take queries from a device work queue, one per warp, as
// warps free up, so a batch ends when its last-started long queries end. A
// query's length is not known before it runs. Two cheap predictors: its ef (a
// search pops at least ef nodes), and its distance to the entry point (where
// every search starts; the farther, the longer the walk to its region). The
// order is by ef, then by that distance, both descending; on the bench's 1M
// batch it shortens the batch by 8 % (ordering by the true pop counts would
// give 24 %). The order changes no result: every query is searched alone.
#include <cub/device/device_radix_sort.cuh>

#include "lqg_host.h"
#include "lqg_internal.h"

namespace lqg {

// key[i] descends with (ef_i, |q_i - decoded entry|^2), so that an ascending
// sort puts the longest-expected queries first; idx[i] = i. One warp per
// query. Without per-query ef: key = ~bits(distance) (non-negative floats
// order as their bits). With it: ~(min(ef, 1023) << 22 | bits(distance) >> 10).
__global__ void entry_distance_kernel(const float* __restrict__ q, int64_t m, uint32_t dim,
                                      const uint8_t* __restrict__ ecode,
                                      const float* __restrict__ params,
                                      const uint32_t* __restrict__ efq, uint32_t* __restrict__ key,
                                      int32_t* __restrict__ idx) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= m) return;  // whole warps
    float s = 0.f;
    for (uint32_t d = lane; d < dim; d += 32) {
        const float dec = fmaf((float)ecode[d], params[2 * d + 1], params[2 * d]);
        const float df = q[(size_t)i * dim + d] - dec;
        s = fmaf(df, df, s);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    if (lane == 0) {
        const uint32_t db = __float_as_uint(s);
        key[i] = efq ? ~((min(efq[i], 1023u) << 22) | (db >> 10)) : ~db;
        idx[i] = (int32_t)i;
    }
}

// Which form of the batch kernel takes a batch of queries with an ef each: the
// latency form if its blocks can start all queries of more than half of the largest
// ef at once and all queries together are the work of at most 1.5 of the largest per
// block. (Such a batch ends when its longest queries do, which the latency form
// finishes sooner, while the short ones leave blocks free.
// us, one-warp against latency form, 100k vectors, k up to 100; ef 32 to 512 in
// equal shares - at 960 dimensions and degree 64, 592 blocks: 1,184 queries 8040 and
// 6402, 2,368 10081 and 7801, 3,552 10284 and 11287; at 128 and 32, 1,184 blocks:
// 2,368 3258 and 2566, 4,736 3405 and 2670, 8,192 3659 and 3638. All at ef 512:
// 888 queries 8473 and 9716; 1,776 at 128 dimensions 3206 and 3288.)
// The latency form's work list is the queries by descending ef, counted into bins in
// one block, in any order within a bin. (A batch that stays with the one-warp form
// pays 10 to 12 us for this kernel and the other form's empty launch up to 2,500
// queries, 20 at 18,000: ef 10, 1,185 queries of 100k x 96 157 against 146 us; with
// the sort above in its place it was 50 to 70.)
__global__ void __launch_bounds__(1024) choose_form_kernel(const uint32_t* __restrict__ efq,
                                                           uint32_t m, uint32_t efmax,
                                                           uint32_t blocks, int32_t* list,
                                                           uint32_t* warp_count,
                                                           uint32_t* latency_count) {
    __shared__ uint32_t start[513];  // by descending ef: count, then first place
    __shared__ uint32_t s_latency;
    const uint32_t t = threadIdx.x, lane = t & 31, rows = (m + 1023) / 1024;
    if (t < 513) start[t] = 0;
    __syncthreads();
    for (uint32_t r = 0; r < rows; ++r) {
        const uint32_t i = r * 1024 + t;
        const uint32_t bin = i < m ? 512 - min(efq[i], efmax) : 513u;
        const unsigned same = __match_any_sync(kFull, bin);
        if (bin < 513 && lane == (uint32_t)__ffs(same) - 1) atomicAdd(&start[bin], __popc(same));
    }
    __syncthreads();
    if (t < 32) {  // 17 bins a lane
        uint32_t n = 0, first = 513;
        uint64_t sum = 0;
        for (uint32_t x = 17 * t; x < min(17 * t + 17, 513u); ++x) {
            n += start[x];
            sum += (uint64_t)start[x] * (512 - x);
            if (start[x] && first == 513) first = x;
        }
        const uint32_t most = 512 - __reduce_min_sync(kFull, first);
        uint32_t many = 0, base = n;
        for (uint32_t x = 17 * t; x < min(17 * t + 17, 513u); ++x)
            if (2 * (512 - x) > most) many += start[x];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, base, o);
            if (lane >= o) base += v;
            sum += __shfl_xor_sync(kFull, sum, o);
        }
        many = __reduce_add_sync(kFull, many);
        base -= n;
        for (uint32_t x = 17 * t; x < min(17 * t + 17, 513u); ++x) {
            const uint32_t c = start[x];
            start[x] = base;
            base += c;
        }
        if (t == 0) {
            const bool latency = many <= blocks && 2 * sum <= 3ull * blocks * most;
            *warp_count = latency ? 0u : m;
            *latency_count = s_latency = latency ? m : 0u;
        }
    }
    __syncthreads();
    if (s_latency == 0) return;
    for (uint32_t r = 0; r < rows; ++r) {
        const uint32_t i = r * 1024 + t;
        const uint32_t bin = i < m ? 512 - min(efq[i], efmax) : 513u;
        const unsigned same = __match_any_sync(kFull, bin);
        const int lead = __ffs(same) - 1;
        uint32_t at = 0;
        if (bin < 513 && (int)lane == lead) at = atomicAdd(&start[bin], __popc(same));
        at = __shfl_sync(kFull, at, lead) + __popc(same & ((1u << lane) - 1u));
        if (bin < 513) list[at] = (int32_t)i;
    }
}

}  // namespace lqg

namespace lqg_host {

// Sizes the work-order buffers for chunks of up to `chunk` queries.
lqg_status ensure_order(Workspace& w, int64_t chunk) {
    lqg_status s;
    if ((s = grow(w.d_okey, w.cap_okey, (size_t)chunk * 2)) != LQG_OK) return s;
    if ((s = grow(w.d_oidx, w.cap_oidx, (size_t)chunk * 2)) != LQG_OK) return s;
    size_t tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (const int32_t*)nullptr, (int32_t*)nullptr, (int)chunk, 0, 32);
    return grow(w.d_otemp, w.cap_otemp, tb);
}

// The work list of queries [0, m) of `queries` (per-query ef efq or NULL):
// longest expected first, sorted on the key's top 16 bits (24 with efq).
lqg_status order_queries(const lqg_index* ix, Workspace& w, const float* queries,
                         const uint32_t* efq, int64_t m, cudaStream_t st, const int32_t** list) {
    uint32_t* kin = w.d_okey;
    uint32_t* kout = w.d_okey + w.cap_okey / 2;
    int32_t* vin = w.d_oidx;
    int32_t* vout = w.d_oidx + w.cap_oidx / 2;
    const int threads = 256;
    const int64_t blocks = (m * 32 + threads - 1) / threads;
    lqg::entry_distance_kernel<<<(unsigned)blocks, threads, 0, st>>>(
        queries, m, ix->dim, ix->d_codes + (size_t)ix->entry * ix->cstride, ix->d_params, efq, kin,
        vin);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "work-order launch");
    size_t tb = w.cap_otemp;
    e = cub::DeviceRadixSort::SortPairs(w.d_otemp, tb, kin, kout, vin, vout, (int)m,
                                        efq ? 8 : 16, 32, st);
    if (e != cudaSuccess) return cuda_fail(e, "work-order sort");
    *list = vout;
    return LQG_OK;
}

// Writes the lengths of the one-warp and the latency form's work lists (one of
// them is 0) for m queries with per-query ef <= efmax, and the latter's list;
// blocks: the latency form's resident blocks. After order_queries, whose list
// stays.
lqg_status choose_form(Workspace& w, const uint32_t* efq, int64_t m, uint32_t efmax,
                       int64_t blocks, cudaStream_t st, const int32_t** list) {
    lqg::choose_form_kernel<<<1, 1024, 0, st>>>(efq, (uint32_t)m, efmax, (uint32_t)blocks,
                                                w.d_oidx, w.d_ctl + kCtlWarpCount,
                                                w.d_ctl + kCtlLatencyCount);
    LQG_CUDA(cudaGetLastError());
    *list = w.d_oidx;
    return LQG_OK;
}

}  // namespace lqg_host
