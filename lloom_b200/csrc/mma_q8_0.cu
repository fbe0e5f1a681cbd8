// Tensor-core skinny product, Q8_0 weights: the kernel instances of this format and their launcher.
#include "gemv_mma.cuh"

namespace lloom {

LLOOM_TU_REGISTER()

cudaError_t launch_mma_q8_0(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream) {
    return launch_mma_format<MmaQ8_0>(p, map, nt, grid_x, grid_y, smem, overlap, stream);
}

}  // namespace lloom
