// Dispatch of the fast search kernel over its pool-size instances.
#include "fast_kernel.cuh"

namespace lqg {

extern template cudaError_t fast_dispatch<1>(const SearchArgs&, int, int, int, size_t, cudaStream_t,
                                             int*);
extern template cudaError_t fast_dispatch<2>(const SearchArgs&, int, int, int, size_t, cudaStream_t,
                                             int*);
extern template cudaError_t fast_dispatch<4>(const SearchArgs&, int, int, int, size_t, cudaStream_t,
                                             int*);
extern template cudaError_t fast_dispatch<8>(const SearchArgs&, int, int, int, size_t, cudaStream_t,
                                             int*);
extern template cudaError_t fast_dispatch<16>(const SearchArgs&, int, int, int, size_t,
                                              cudaStream_t, int*);

static cudaError_t dispatch(const SearchArgs& a, int E, int degw, int warps, int blocks,
                            size_t smem, cudaStream_t st, int* occ) {
    switch (E) {
        case 1: return fast_dispatch<1>(a, degw, warps, blocks, smem, st, occ);
        case 2: return fast_dispatch<2>(a, degw, warps, blocks, smem, st, occ);
        case 4: return fast_dispatch<4>(a, degw, warps, blocks, smem, st, occ);
        case 8: return fast_dispatch<8>(a, degw, warps, blocks, smem, st, occ);
        case 16: return fast_dispatch<16>(a, degw, warps, blocks, smem, st, occ);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_fast(const SearchArgs& a, int E, int degw, int warps, int blocks,
                        cudaStream_t st) {
    return dispatch(a, E, degw, warps, blocks, fast_smem_bytes(a.dim, a.deg, a.vbits, a.sbits, warps), st,
                    nullptr);
}

int fast_occupancy(int E, int degw, int warps, uint32_t dim, uint32_t vbits, uint32_t sbits) {
    int occ = 0;
    SearchArgs a{};
    if (dispatch(a, E, degw, warps, 0, fast_smem_bytes(dim, 32u * degw, vbits, sbits, warps),
                 nullptr, &occ) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return occ;
}

}  // namespace lqg
