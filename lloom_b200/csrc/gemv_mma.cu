// Activation images of the tensor-core skinny product (gemv_mma.cuh).
#include "gemv_mma.cuh"

namespace lloom {

LLOOM_TU_REGISTER()

// code offset of the weights, taken out through the accumulator start (Q4_0: nibble - 8, Q5_0: code - 16)
static int code_offset(int w_dtype) { return w_dtype == LLOOM_Q4_0 ? 8 : w_dtype == LLOOM_Q5_0 ? 16 : 0; }

cudaError_t launch_quantize_image(int w_dtype, const void *x, int x_type, uint8_t *img, int64_t m, int64_t k, int tiles, int group_nt,
                                  bool overlap, cudaStream_t stream) {
    const int rows = image_rows(m);
    const int64_t warps = (int64_t)tiles * rows * ((k + 255) / 256);
    return launch_early(quantize_image_kernel, (unsigned)ceil_div64(warps, kQuantThreads / 32), kQuantThreads, 0, overlap, stream, x, x_type, img, image_kind(w_dtype),
                        code_offset(w_dtype), image_unit_bytes(w_dtype, rows), (int)m, (int)k, tiles, group_nt, rows);
}

cudaError_t launch_blocks_image(int w_dtype, const void *act, uint8_t *img, int64_t m, int64_t k, int group_nt, cudaStream_t stream) {
    const int64_t items = m * (k / 32) * 8;
    const unsigned grid = (unsigned)(ceil_div64(items, 256) < 4096 ? ceil_div64(items, 256) : 4096);
    blocks_to_image_kernel<<<grid, 256, 0, stream>>>((const uint8_t *)act, img, image_kind(w_dtype), code_offset(w_dtype),
                                                     image_unit_bytes(w_dtype, image_rows(m)), (int)m, (int)k, group_nt, image_rows(m));
    return cudaGetLastError();
}

}  // namespace lloom
