// dp4a decode GEMV, Q4K weights: the kernel instances of this format and their launcher.
#include "gemv.cuh"

namespace lloom {

LLOOM_TU_REGISTER()

cudaError_t launch_gemv_dp4a_q4k(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream) {
    return launch_gemv_format<FmtQ4K>(p, grid, smem, overlap, rw, stream);
}

}  // namespace lloom
