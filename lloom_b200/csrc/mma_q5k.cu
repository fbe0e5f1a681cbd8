// Tensor-core skinny product, Q5K weights: the kernel instances of this format and their launcher.
#include "gemv_mma.cuh"

namespace lloom {

LLOOM_TU_REGISTER()

cudaError_t launch_mma_q5k(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream) {
    return launch_mma_format<MmaQ5K>(p, map, nt, grid_x, grid_y, smem, overlap, stream);
}

}  // namespace lloom
