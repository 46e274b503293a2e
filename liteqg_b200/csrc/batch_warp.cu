// Batched-acceptance search kernel, one warp per query: an instance per degree
// word count.
#include "batch_kernel.cuh"

namespace lqg {

cudaError_t launch_batch(const SearchArgs& a, const ReplayArgs& ra, int degw, int warps, int blocks,
                         cudaStream_t st, int* occ) {
    switch (degw) {
        case 1: return batch_run<1>(a, ra, warps, blocks, st, occ);
        case 2: return batch_run<2>(a, ra, warps, blocks, st, occ);
        case 3: return batch_run<3>(a, ra, warps, blocks, st, occ);
        case 4: return batch_run<4>(a, ra, warps, blocks, st, occ);
        default: return cudaErrorInvalidValue;
    }
}

bool batch_replays_in_place_host(uint32_t deg, uint32_t vbits, uint32_t scap, uint32_t acap,
                                 uint32_t rcap) {
    return batch_replays_in_place(deg, vbits, scap, acap, rcap);
}

}  // namespace lqg
