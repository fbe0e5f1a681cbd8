// Launch parameters and shared-memory sizing of the decode GEMV kernels: the part of gemv.cuh / gemv_mma.cuh
// that the host-side planner (lloom_b200.cu) and the kernels' translation units both need.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/lloom_b200.h"

namespace lloom {

constexpr int kQ8KUnitStride = 256 + 16;
constexpr int kQ8_0UnitStride = 64 + 16;
constexpr int kMaxStages = 8;
constexpr int kMaxPeers = 8;  // GPUs of one node
constexpr int kMaxGroup = LLOOM_B200_MAX_GROUP;  // weight matrices one grouped launch streams

__host__ __device__ inline int64_t elem_bytes(int type) { return type == LLOOM_F32 ? 4 : 2; }
__host__ __device__ inline int64_t round16(int64_t v) { return (v + 15) / 16 * 16; }

// Activation planes in shared memory, built once per CTA (layouts: gemv.cuh).  Formats dotted with Q8_0
// activations work on units of 64 elements, the k-quants on 256-element superblocks.
__host__ __device__ inline bool act_is_q8_0(int w_dtype) {
    return w_dtype == LLOOM_Q8_0 || w_dtype == LLOOM_Q4_0 || w_dtype == LLOOM_Q5_0;
}
__host__ __device__ inline int64_t act_qs_bytes(int w_dtype, int64_t m, int64_t k) {
    return act_is_q8_0(w_dtype) ? m * (k / 64) * kQ8_0UnitStride : m * (k / 256) * kQ8KUnitStride;
}
__host__ __device__ inline int64_t act_plane_bytes(int w_dtype, int64_t m, int64_t k) {
    const int64_t qs = act_qs_bytes(w_dtype, m, k);
    const int64_t d = act_is_q8_0(w_dtype) ? m * (k / 32) * 4 : m * (k / 256) * 4;
    const int64_t sums = act_is_q8_0(w_dtype) ? (w_dtype == LLOOM_Q8_0 ? 0 : m * (k / 32) * 4)
                                              : (w_dtype == LLOOM_Q6_K ? m * (k / 16) * 2 : m * (k / 32) * 2);
    return round16(qs) + round16(d) + round16(sums);
}

struct GemvParams {
    const uint8_t *w;    // canonical blocks, 16-byte aligned
    const uint8_t *act;  // canonical activation blocks [m][k/block] (used when x == nullptr)
    const void *x;       // activations [m][k] of type x_type, 16-byte aligned: quantized in the prologue (fused forward)
    float *y;            // outputs of type y_type (anything but f32 only where there is one matrix and a plain store)
    int x_type, y_type;
    int64_t ldy;
    int64_t row_bytes;
    int64_t w_bytes;  // n * row_bytes
    int n, k, m;
    int w_dtype;
    int n_cwarps;      // consumer warps; blockDim.x = 32 * (n_cwarps + 1)
    int lpr_log2;      // lanes per row = 1 << lpr_log2 (a warp handles 32 / lanes-per-row row groups)
    int stages;
    int stage_bytes;   // multiple of 128
    int act_bytes;     // multiple of 16
    int nchunks;         // dp4a kernel: pieces a row is cut into, each a stage's worth (1: whole rows)
    int chunk_units;     // dp4a kernel, nchunks > 1: units (superblocks / pairs of 32-element blocks) of a row per piece
    int unit_bytes;      // dp4a kernel: bytes of a unit
    // Tensor-core kernel (gemv_mma.cuh).
    const uint8_t *img;   // activation image in global memory, or null: quantized (x) or rearranged (act) in the prologue
    int img_unit;         // bytes of a unit
    int group_nt;         // activation tiles a CTA works on (blockIdx.y: group of them)
    int nsb;              // 256-element superblocks of a row (the last one may be short in the 32-element formats)
    int split;            // S: superblocks per stage, one per slot warp
    int second;           // two sums per warp (S = 4): bytes from a warp's first superblock of a slice to its second; else 0
    int col_parts;        // TN: warps that share the activation tiles
    int tile_rows_cta;    // TR * 16: rows per tile group
    int slice_sb;         // superblocks of a row per stage, a multiple of S
    int slice_bytes;      // their bytes
    int row_pitch;        // bytes between weight rows inside a stage (a box is 16 rows of it)
    int boxes;            // TMA boxes per tile and stage; 0: a bulk copy per row
    int box_sb, box_step; // superblocks of a box, and its width without the padding in elements of 8 bytes
    int box_bytes;
    int act_stream;       // activations travel with the stages (else they are resident: act_bytes)
    int act_stage_off;    // where in a stage
    int red_bytes;        // partial sums
    int act_copy;         // bytes of a resident image
    // Fused gather: when n_peers > 0 every output value goes to the same place in each of these buffers (this GPU's
    // own and its peers', mapped into this process) instead of `y`, so the row-sharded forward needs no separate
    // all-gather: the stores cross NVLink while the rest of the rows are still being computed.
    int n_peers;
    // Fused gather with staging: bytes of the shared-memory area (after the activation planes) that collects the
    // CTA's output rows, [m][out_pitch] floats; the CTA writes them to the peers in whole lines when it is done.
    // 0: every value goes out on its own.
    int out_bytes;
    int out_pitch;
    // Block on the store (the reference's MvStore, lloom-tensor/src/quantized/mod.rs:1668-1696):
    // 0 plain, 1 silu(W.x), 2 dst <- dst * (W.x).
    int store_mode;
    // Fused gather, barrier folded into the GEMV (publish != 0): the last CTA to finish advances this GPU's call
    // counter and stores it in slot [peer_rank] of every GPU's flag array (lloom_b200_qmatmul_fwd_gather_sync).
    // wait_flags != nullptr: the activations came out of an earlier fused gather whose flag array (this GPU's)
    // this is; the kernel waits for all `wait_peers` slots to reach that gather's count before it reads them.
    unsigned int *peer_flags[kMaxPeers];
    const unsigned int *wait_flags;
    int wait_peers;
    int publish;
    int peer_rank;
    float *y_peer[kMaxPeers];
    // Grouped launch (n_group > 1): matrices of one dtype and k that share the activations, streamed by one launch.
    // The kernel walks the concatenation of their rows; `n` is the total.  Matrix g: rows [goff[g], goff[g+1]).
    int n_group;
    const uint8_t *gw[kMaxGroup];
    float *gy[kMaxGroup];
    int64_t gldy[kMaxGroup];
    int goff[kMaxGroup + 1];
    int gstore[kMaxGroup];
    // Routed experts (moe_ids != nullptr, grouped launches only): matrix g is expert moe_ids[g] of the stacked
    // tensor at `w` (every expert has as many rows as the group's matrices); the ids are device data, read after the
    // stream predecessor is done.
    const uint32_t *moe_ids;
    int moe_experts;
    int moe_id_words;  // 32-bit words per id: 1, or 2 for 64-bit ids (the low word counts)
    // blockIdx.y counts items (a token's experts, or one product), the launch's first being item0 of its activation row:
    // item i reads row (item0 + i) / x_per
    unsigned x_per, item0;
    // What a launch costs on the host depends on the size of this block: a call of one row [1024, 4096], host-bound, takes 3.45 us
    // with 664 or 672 bytes and 3.70 to 3.75 with 656, 680 or 704 (medians of four processes each on one machine).
    int pad[4];
};
static_assert(sizeof(GemvParams) == 672, "see pad");

// ---- tensor-core kernel (gemv_mma.cuh) ----
constexpr int kMmaTileRows = 16;
constexpr int kMmaWarps = 16;          // most consumer warps
constexpr int kMmaStages = 8;
constexpr int kMmaBarBytes = 256;      // full / empty barriers, one for the resident activations, one flag
constexpr int kMmaSlack = 128;         // word-wise reads may run a few bytes past the last stage
constexpr int kMmaMaxTeams = 7;        // two named barriers each
enum { kImgK, kImgQ6K, kImg32, kImgSplit };  // orders of the activation codes

__host__ __device__ inline int image_kind(int w_dtype) {
    switch (w_dtype) {
    case LLOOM_Q6_K: return kImgQ6K;
    case LLOOM_Q8_0: return kImg32;
    case LLOOM_Q4_0: case LLOOM_Q5_0: return kImgSplit;
    }
    return kImgK;
}
// rows of an activation tile: eight, or a single row on its own
__host__ __device__ inline int image_rows(int64_t m) { return m == 1 ? 1 : 8; }
// bytes of a unit: a tile of activation rows x 256 elements
__host__ __device__ inline int image_unit_bytes(int w_dtype, int rows) {
    const int kind = image_kind(w_dtype);
    const int per_row = 256 + (kind == kImg32 ? 32 : kind == kImgSplit ? 64 : 36);
    return (per_row * rows + 15) / 16 * 16;
}

// Smallest pitch in bytes (a multiple of 16, >= bytes) that is an odd multiple of `unit` (4 or 8) 32-bit words.
__host__ __device__ inline int64_t bank_pitch(int64_t bytes, int unit) {
    int64_t q = (bytes + 4 * unit - 1) / (4 * unit);
    if (q % 2 == 0) ++q;
    return q * unit * 4;
}

// ---- launchers exported by the kernels' translation units ----
// dp4a GEMV, one unit per weight format.  rw: rows per lane (1 or 2).
cudaError_t launch_gemv_dp4a_q8_0(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream);
cudaError_t launch_gemv_dp4a_q4k(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream);
cudaError_t launch_gemv_dp4a_q6k(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream);
cudaError_t launch_gemv_dp4a_q5k(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream);
cudaError_t launch_gemv_dp4a_q4_0(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream);
cudaError_t launch_gemv_dp4a_q5_0(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream);
// tensor-core kernel, one unit per weight format.  nt: activation tiles per warp (1..3)
cudaError_t launch_mma_q8_0(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream);
cudaError_t launch_mma_q4k(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream);
cudaError_t launch_mma_q6k(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream);
cudaError_t launch_mma_q5k(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream);
cudaError_t launch_mma_q4_0(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream);
cudaError_t launch_mma_q5_0(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream);
// The activation image of m rows in `tiles` (whole groups of group_nt) tiles: from values, or from canonical blocks.
cudaError_t launch_quantize_image(int w_dtype, const void *x, int x_type, uint8_t *img, int64_t m, int64_t k, int tiles, int group_nt,
                                  bool overlap, cudaStream_t stream);
cudaError_t launch_blocks_image(int w_dtype, const void *act, uint8_t *img, int64_t m, int64_t k, int group_nt, cudaStream_t stream);

}  // namespace lloom
