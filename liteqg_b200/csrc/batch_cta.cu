// Batched-acceptance search kernel, latency form (one query per block: a merging
// warp and expanding warps), for small batches.
#include "batch_kernel.cuh"

namespace lqg {

cudaError_t launch_batch_cta(const SearchArgs& a, const ReplayArgs& ra, int degw, int blocks,
                             cudaStream_t st, int* occ) {
    switch (degw) {
        case 1: return batch_run<1, true>(a, ra, 1, blocks, st, occ);
        case 2: return batch_run<2, true>(a, ra, 1, blocks, st, occ);
        case 3: return batch_run<3, true>(a, ra, 1, blocks, st, occ);
        case 4: return batch_run<4, true>(a, ra, 1, blocks, st, occ);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace lqg
