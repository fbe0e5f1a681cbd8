// Prefill GEMM (more than 128 rows, or fewer against a prebuilt image): the tcgen05 kernels' translation unit -- planning
// of the operand images, their build kernels and the launches.  Q4_K, Q5_K: gemm_q4k.cuh; the others: gemm_planes.cuh.
#include "gemm.h"

#include <mutex>

#include "gemm_planes.cuh"
#include "gemv_params.h"

namespace lloom {

LLOOM_TU_REGISTER()

namespace {

using CfgQ8_0 = PlanesCfg<32, 1, 128>;
using CfgQ6K = PlanesCfg<256, 2, 256>;
using CfgQ6KSmall = PlanesCfg<256, 2, 128>;

// Activation rows per tile of the Q6_K GEMM for m rows against n_tiles x 128 weight rows.  A 256-row tile does more per byte
// it reads from shared memory: a 128-row tile takes kSmallTile of its time, not half (29.2 against 51.6 us a round over
// the SMs at k = 4096: 13 small rounds take 379 us where 7 large ones take 361).  The shape whose rounds take less time is
// run ([4096, 14336] with 512 rows, image prebuilt, 64 large tiles or 128 small ones on 148 SMs: 162 -> 110 us in a loop over
// two warm matrices, 165 -> 131 us with inputs that change from call to call); both give the same bits.
constexpr double kSmallTile = 0.57;
int q6k_bm(int64_t m, int64_t n_tiles, int sms) {
    const int64_t big = ((m + 255) / 256 * n_tiles + sms - 1) / sms, small = ((m + 127) / 128 * n_tiles + sms - 1) / sms;
    return (double)small * kSmallTile < (double)big ? CfgQ6KSmall::kBM : CfgQ6K::kBM;
}

// Weight images of more than this are built and consumed slab by slab (whole 128-row tiles), so that the
// caller's workspace stays bounded whatever the matrix (a Q6_K lm_head image is 2.1 GB).
constexpr int64_t kSlabImageBytes = 256ll << 20;

struct OnceSmem {  // dynamic shared memory opt-in, per device
    std::mutex mu;
    bool done[64] = {false};
};

template <class Kern>
cudaError_t opt_in_smem(Kern kern, OnceSmem &st, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(st.mu);
    if (st.done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) st.done[dev] = true;
    return e;
}

int64_t image_bytes_for_rows(int w_dtype, int64_t rows, int64_t k) {
    switch (w_dtype) {
    case LLOOM_Q4_K:
    case LLOOM_Q5_K: return gemm_weight_layout(rows, k).total;
    case LLOOM_Q8_0:
    case LLOOM_Q4_0:
    case LLOOM_Q5_0: return planes_weight_bytes(rows, k, 1);
    case LLOOM_Q6_K: return planes_weight_bytes(rows, k, 2);
    }
    return 0;
}

int64_t act_image_bytes(int w_dtype, int64_t m, int64_t k) {
    switch (w_dtype) {
    case LLOOM_Q4_K:
    case LLOOM_Q5_K: return gemm_act_layout(m, k).total;
    case LLOOM_Q8_0:
    case LLOOM_Q4_0:
    case LLOOM_Q5_0: return planes_act_layout(m, k, 32, CfgQ8_0::kBM).total;
    case LLOOM_Q6_K: return planes_act_layout(m, k, 256, CfgQ6K::kBM).total;  // of both tile shapes the larger
    }
    return 0;
}

template <int DTYPE>
cudaError_t expand_planes(const uint8_t *w, int64_t rows, int64_t k, uint8_t *image, bool beside, cudaStream_t stream) {
    const int64_t nt = (rows + kGemmBN - 1) / kGemmBN, row_bytes = k / lloom_b200_block_elems(DTYPE) * lloom_b200_block_bytes(DTYPE);
    return launch_early(planes_expand_kernel<DTYPE>, (unsigned)(nt * (k / 128) * 4), 256, 0, beside, stream, w, row_bytes, (int)rows, (int)k, image);
}

// `beside`: the stream predecessor is this call's activation side, started after everything before the call was done; the
// image may be built while it runs.
cudaError_t build_image(int w_dtype, const uint8_t *w, int64_t rows, int64_t k, uint8_t *image, bool beside, cudaStream_t stream) {
    const unsigned grid = (unsigned)((rows + kGemmBN - 1) / kGemmBN * (k / 256) * 4);
    switch (w_dtype) {
    case LLOOM_Q4_K: return launch_early(gemm_expand_kernel<false>, grid, 256, 0, beside, stream, w, (int)rows, (int)k, image);
    case LLOOM_Q5_K: return launch_early(gemm_expand_kernel<true>, grid, 256, 0, beside, stream, w, (int)rows, (int)k, image);
    case LLOOM_Q8_0: return expand_planes<LLOOM_Q8_0>(w, rows, k, image, beside, stream);
    case LLOOM_Q4_0: return expand_planes<LLOOM_Q4_0>(w, rows, k, image, beside, stream);
    case LLOOM_Q5_0: return expand_planes<LLOOM_Q5_0>(w, rows, k, image, beside, stream);
    case LLOOM_Q6_K: return expand_planes<LLOOM_Q6_K>(w, rows, k, image, beside, stream);
    }
    return cudaErrorInvalidValue;
}

template <class Cfg>
cudaError_t launch_planes(const PlanesParams &p, cudaStream_t stream) {
    static OnceSmem once;
    cudaError_t e = opt_in_smem(gemm_planes_kernel<Cfg>, once, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    return launch_early(gemm_planes_kernel<Cfg>, (unsigned)(p.n_tiles * p.m_tiles), Cfg::kThreads, Cfg::kSmemBytes, true, stream, p);
}

}  // namespace

bool gemm_supported(int w_dtype, int64_t m, int64_t k, int max_smem) {
    if (m <= 8) return false;
    switch (w_dtype) {
    case LLOOM_Q4_K:
    case LLOOM_Q5_K: return k % 256 == 0 && kGemmSmemBytes <= max_smem;
    case LLOOM_Q6_K: return k % 256 == 0 && CfgQ6K::kSmemBytes <= max_smem && CfgQ6KSmall::kSmemBytes <= max_smem;
    case LLOOM_Q8_0:
    case LLOOM_Q4_0:
    case LLOOM_Q5_0: return k % 128 == 0 && CfgQ8_0::kSmemBytes <= max_smem;  // a pipeline stage is 128 of K
    }
    return false;
}

int64_t gemm_weight_image_bytes(int w_dtype, int64_t n, int64_t k) { return image_bytes_for_rows(w_dtype, n, k); }

int64_t gemm_slab_rows(int w_dtype, int64_t n, int64_t k) {
    const int64_t per_tile = image_bytes_for_rows(w_dtype, kGemmBN, k);
    if (per_tile <= 0) return 0;
    int64_t tiles = kSlabImageBytes / per_tile;
    if (tiles < 1) tiles = 1;
    const int64_t all = (n + kGemmBN - 1) / kGemmBN;
    return (tiles < all ? tiles : all) * kGemmBN;
}

int64_t gemm_scratch_bytes(int w_dtype, int64_t m, int64_t n, int64_t k, bool have_image) {
    if (m <= 8) return 0;
    const int64_t act = act_image_bytes(w_dtype, m, k);
    if (act <= 0) return 0;
    if (have_image) return act;
    const int64_t rows = gemm_slab_rows(w_dtype, n, k);
    return act + (image_bytes_for_rows(w_dtype, rows, k) + 255) / 256 * 256;
}

cudaError_t gemm_weight_image_build(int w_dtype, const void *w, int64_t n, int64_t k, void *image, cudaStream_t stream) {
    return build_image(w_dtype, (const uint8_t *)w, n, k, (uint8_t *)image, false, stream);
}

cudaError_t gemm_forward(int w_dtype, const void *w_blocks, const void *w_image, const void *act, const void *x, int x_type, void *y,
                         int y_type, int64_t m, int64_t n, int64_t k, int64_t ldy, void *scratch, cudaStream_t stream) {
    if ((act == nullptr) == (x == nullptr)) return cudaErrorInvalidValue;
    const uint8_t *w = (const uint8_t *)w_blocks;
    uint8_t *act_img = (uint8_t *)scratch;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int64_t slab = w_image ? n : gemm_slab_rows(w_dtype, n, k);
    const int bm = w_dtype == LLOOM_Q6_K ? q6k_bm(m, ((slab < n ? slab : n) + kGemmBN - 1) / kGemmBN, sms) : kGemmBM;
    const int64_t mt = (m + bm - 1) / bm;
    // activation side, once per call
    const bool q4k_frame = w_dtype == LLOOM_Q4_K || w_dtype == LLOOM_Q5_K;
    const bool q8_0_frame = w_dtype == LLOOM_Q8_0 || w_dtype == LLOOM_Q4_0 || w_dtype == LLOOM_Q5_0;
    if (q4k_frame && x) {
        gemm_prep_f32_kernel<<<(unsigned)(mt * kGemmBM * (k / 256) / 8), 256, 0, stream>>>(x, x_type, (int)m, (int)k, act_img);
    } else if (q4k_frame) {
        gemm_prep_kernel<<<(unsigned)(mt * (k / 256) * 4), 256, 0, stream>>>((const uint8_t *)act, (int)m, (int)k, act_img);
    } else if (q8_0_frame && x) {
        planes_prep_f32_kernel<true, CfgQ8_0::kBM><<<(unsigned)(mt * CfgQ8_0::kBM * ((k + 255) / 256) / 8), 256, 0, stream>>>(x, x_type, (int)m, (int)k, act_img);
    } else if (w_dtype == LLOOM_Q6_K && x) {
        if (bm == CfgQ6K::kBM)
            planes_prep_f32_kernel<false, CfgQ6K::kBM><<<(unsigned)(mt * CfgQ6K::kBM * (k / 256) / 8), 256, 0, stream>>>(x, x_type, (int)m, (int)k, act_img);
        else
            planes_prep_f32_kernel<false, CfgQ6KSmall::kBM><<<(unsigned)(mt * CfgQ6KSmall::kBM * (k / 256) / 8), 256, 0, stream>>>(x, x_type, (int)m, (int)k, act_img);
    } else if (q8_0_frame) {
        planes_prep_kernel<true, CfgQ8_0::kBM><<<(unsigned)(mt * (k / 64)), CfgQ8_0::kBM, 0, stream>>>((const uint8_t *)act, (int)m, (int)k, act_img);
    } else if (w_dtype == LLOOM_Q6_K) {
        if (bm == CfgQ6K::kBM)
            planes_prep_kernel<false, CfgQ6K::kBM><<<(unsigned)(mt * (k / 64)), CfgQ6K::kBM, 0, stream>>>((const uint8_t *)act, (int)m, (int)k, act_img);
        else
            planes_prep_kernel<false, CfgQ6KSmall::kBM><<<(unsigned)(mt * (k / 64)), CfgQ6KSmall::kBM, 0, stream>>>((const uint8_t *)act, (int)m, (int)k, act_img);
    } else {
        return cudaErrorInvalidValue;
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int64_t row_bytes = k / lloom_b200_block_elems(w_dtype) * lloom_b200_block_bytes(w_dtype);
    uint8_t *slab_img = act_img + act_image_bytes(w_dtype, m, k);
    for (int64_t row0 = 0; row0 < n; row0 += slab) {
        const int64_t rows = n - row0 < slab ? n - row0 : slab;
        const uint8_t *w_slab = w + row0 * row_bytes;
        const uint8_t *img = (const uint8_t *)w_image;
        if (!img) {  // later slabs: the previous slab's GEMM has read the buffer before this build overwrites it
            e = build_image(w_dtype, w_slab, rows, k, slab_img, row0 == 0, stream);
            if (e != cudaSuccess) return e;
            img = slab_img;
        }
        const int n_tiles = (int)((rows + kGemmBN - 1) / kGemmBN);
        if (q4k_frame) {
            static OnceSmem once;
            e = opt_in_smem(gemm_q4k_kernel, once, kGemmSmemBytes);
            if (e != cudaSuccess) return e;
            GemmParams p;
            p.w = w_slab;
            p.act_img = act_img;
            p.w_img = img;
            p.y = (uint8_t *)y + row0 * elem_bytes(y_type);
            p.y_type = y_type;
            p.ldy = ldy;
            p.row_bytes = row_bytes;
            p.m = (int)m;
            p.n = (int)rows;
            p.k = (int)k;
            p.n_tiles = n_tiles;
            p.m_tiles = (int)mt;
            p.blk_bytes = (int)lloom_b200_block_bytes(w_dtype);
            const int64_t tiles = n_tiles * mt;
            e = launch_early(gemm_q4k_kernel, (unsigned)(tiles < sms ? tiles : sms), kQ4kThreads, kGemmSmemBytes, true, stream, p);
        } else {
            PlanesParams p;
            p.w = w_slab;
            p.act_img = act_img;
            p.w_img = img;
            p.y = (uint8_t *)y + row0 * elem_bytes(y_type);
            p.y_type = y_type;
            p.ldy = ldy;
            p.row_bytes = row_bytes;
            p.m = (int)m;
            p.n_end = (int)rows;
            p.k = (int)k;
            p.n_tiles = n_tiles;
            p.m_tiles = (int)mt;
            if (q8_0_frame) {
                p.scale_stride = (int)lloom_b200_block_bytes(w_dtype);  // the f16 scale opens every 32-element block
                p.scale_off = 0;
                e = launch_planes<CfgQ8_0>(p, stream);
            } else {
                p.scale_stride = Q6K_BYTES;
                p.scale_off = 208;
                e = bm == CfgQ6K::kBM ? launch_planes<CfgQ6K>(p, stream) : launch_planes<CfgQ6KSmall>(p, stream);
            }
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace lloom
