// Per-node and per-list-slot sums of the integer distance bound
// (sq8_filter.cuh): nsum[i] = sum (scale code)^2 over node i's code row, and
// esum[i][j] = nsum[nbrs[i][j]], so that a popped node's list brings its
// neighbours' sums in the same coalesced read as their ids (a gather per
// neighbour would cost a 32-byte sector each).
#include <algorithm>
#include <mutex>

#include "lqg_host.h"
#include "lqg_internal.h"

namespace lqg {

// One warp per row; rows are padded to 16 bytes, the padding is skipped.
__global__ void node_sum_kernel(const uint8_t* __restrict__ codes, const float* __restrict__ params,
                                uint64_t n, uint32_t dim, uint32_t cstride,
                                float* __restrict__ nsum) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t i = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
         i += warps) {
        double s = 0.0;
        for (uint32_t d = 4 * lane; d < dim; d += 128) {
            const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(codes + i * cstride + d));
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (d + t < dim) {
                    const double x = (double)params[2 * (d + t) + 1] * (double)((w >> (8 * t)) & 255u);
                    s += x * x;
                }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
        if (lane == 0) nsum[i] = (float)s;
    }
}

__global__ void edge_sum_kernel(const uint32_t* __restrict__ nbrs, const float* __restrict__ nsum,
                                uint64_t edges, float* __restrict__ esum) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < edges;
         e += (uint64_t)gridDim.x * blockDim.x)
        esum[e] = nsum[nbrs[e]];
}

// One warp per list: does any id stand in two of its slots?
__global__ void repeated_id_kernel(const uint32_t* __restrict__ nbrs, uint64_t n, uint32_t deg,
                                   uint32_t* __restrict__ found) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t i = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
         i += warps) {
        const uint32_t* l = nbrs + i * deg;
        bool same = false;
        for (uint32_t w = 0; w < deg; w += 32) {
            const uint32_t v = l[w + lane];
            for (uint32_t e = w; e < deg; e += 32) {  // slots of this word and the later ones
                const uint32_t x = l[e + lane];
#pragma unroll
                for (int o = 0; o < 32; ++o)  // slot (lane + o) % 32 of word e
                    same |= (e > w || o > 0) && v == __shfl_sync(kFull, x, (lane + o) & 31);
            }
        }
        if (same) *found = 1u;
    }
}

}  // namespace lqg

namespace lqg_host {

namespace {

// The indexes that hold sums. Lock order: the list, then an index's sums.
struct Holders {
    std::mutex mu;
    std::vector<lqg_index*> list;
};
Holders& holders() {
    static Holders* h = new Holders;  // outlives every index
    return *h;
}

// Frees ix's sums; with the list and the sums locked.
void free_sums(Holders& h, lqg_index* ix) {
    dfree(ix->d_nsum);
    dfree(ix->d_esum);
    ix->captured = false;
    h.list.erase(std::remove(h.list.begin(), h.list.end(), ix), h.list.end());
}

}  // namespace

void drop_sums(lqg_index* ix) {
    Holders& h = holders();
    std::lock_guard<std::mutex> lk(h.mu);
    std::unique_lock<std::shared_mutex> l(ix->sums_mu);
    free_sums(h, ix);
}

bool give_back_sums(lqg_index* ix) {
    Holders& h = holders();
    std::lock_guard<std::mutex> lk(h.mu);
    lqg_index* from = nullptr;  // its own rather than another's
    for (lqg_index* x : h.list)
        if (x->device == ix->device && !x->captured && (!from || x == ix)) from = x;
    if (!from) return false;
    DeviceScope ds(from->device);
    std::unique_lock<std::shared_mutex> l(from->sums_mu);  // no further call reads them
    if (from->captured || ds.err != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    free_sums(h, from);
    return true;
}

lqg_status check_distinct(lqg_index* ix, cudaStream_t st) {
    ix->distinct = 0;
    uint32_t* d = nullptr;
    if (cudaMalloc(&d, sizeof(uint32_t)) != cudaSuccess) {
        cudaGetLastError();
        return fail(LQG_ERR_NOMEM, "device allocation of the index failed");
    }
    uint32_t found = 1;
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess) {
        lqg::repeated_id_kernel<<<8 * ix->num_sms, 256, 0, st>>>(ix->d_nbrs, ix->n, ix->deg, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&found, d, sizeof(found), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) return cuda_fail(e, "neighbour list check");
    ix->distinct = found ? 0u : 1u;
    return LQG_OK;
}

lqg_status filter_node_sums(lqg_index* ix, cudaStream_t st) {
    std::shared_lock<std::shared_mutex> lk(ix->sums_mu);
    if (!ix->d_nsum || !ix->d_esum) return LQG_OK;
    lqg::node_sum_kernel<<<8 * ix->num_sms, 256, 0, st>>>(ix->d_codes, ix->d_params, ix->n, ix->dim,
                                                          ix->cstride, ix->d_nsum);
    LQG_CUDA(cudaGetLastError());
    return LQG_OK;
}

lqg_status filter_edge_sums(lqg_index* ix, cudaStream_t st) {
    std::shared_lock<std::shared_mutex> lk(ix->sums_mu);
    if (!ix->d_nsum || !ix->d_esum) return LQG_OK;
    lqg::edge_sum_kernel<<<8 * ix->num_sms, 256, 0, st>>>(ix->d_nbrs, ix->d_nsum,
                                                          ix->n * ix->deg, ix->d_esum);
    LQG_CUDA(cudaGetLastError());
    return LQG_OK;
}

void filter_alloc(lqg_index* ix) {
    Holders& h = holders();
    std::lock_guard<std::mutex> lk(h.mu);
    std::unique_lock<std::shared_mutex> l(ix->sums_mu);
    free_sums(h, ix);
    try {
        h.list.push_back(ix);
    } catch (...) {
        return;  // no room for the list: no sums
    }
    if (cudaMalloc(&ix->d_nsum, ix->n * sizeof(float)) == cudaSuccess &&
        cudaMalloc(&ix->d_esum, ix->n * ix->deg * sizeof(float)) == cudaSuccess)
        return;
    cudaGetLastError();
    free_sums(h, ix);
}

void filter_done(lqg_index* ix) {
    std::unique_lock<std::shared_mutex> lk(ix->sums_mu);
    dfree(ix->d_nsum);
}

}  // namespace lqg_host
