// C ABI of the library (see include/lloom_b200.h): argument checks, launch planning and dispatch.  The kernels live
// in translation units of their own (gemv_*.cu, gemv_mma.cu, gemm.cu); this one holds the small ones (activation
// quantizers, dequantize, the peer barrier).  No entry point on the forward path allocates, frees or synchronises.
#include "common.cuh"
#include "dequant.cuh"
#include "forward.h"
#include "gemm.h"
#include "gemv_params.h"
#include "quantize_act.cuh"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

namespace lloom {

LLOOM_TU_REGISTER()

// ---- translation-unit registry: every unit has its own device-side status word and wait limit ----
namespace {
struct TuRegistry {
    std::mutex mu;
    std::vector<TuHooks> hooks;
};
TuRegistry &tu_registry() {
    static TuRegistry r;
    return r;
}
}  // namespace

void register_tu(const TuHooks &hooks) {
    TuRegistry &r = tu_registry();
    std::lock_guard<std::mutex> lock(r.mu);
    r.hooks.push_back(hooks);
}

static thread_local int t_last_cuda_error = 0;

static int launch_status(cudaError_t e) {
    if (e == cudaSuccess) return LLOOM_OK;
    t_last_cuda_error = (int)e;
    return LLOOM_ERR_LAUNCH;
}

static bool supported_weight(int dtype) {
    switch (dtype) {
    case LLOOM_Q8_0: case LLOOM_Q4_K: case LLOOM_Q6_K: case LLOOM_Q4_0: case LLOOM_Q5_0: case LLOOM_Q5_K: return true;
    }
    return false;
}

struct DeviceInfo {
    int sm_count = 0;
    int max_smem_optin = 0;   // per block
    int smem_per_sm = 0;      // per multiprocessor
    int smem_reserved = 0;    // per block, taken by the driver
    int cc_major = 0;
    bool ok = false;
};

// Launch overlap (programmatic dependent launch): lloom_b200_set_launch_overlap.
static std::atomic<int> g_launch_overlap{-1};
int launch_overlap() { return g_launch_overlap.load(std::memory_order_relaxed); }

// Per-device attributes, queried once (the reference caches the same facts, fast_mmq.rs device-info cache).
static int device_info(DeviceInfo &out) {
    static std::mutex mu;
    static DeviceInfo cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LLOOM_ERR_DEVICE;
    std::lock_guard<std::mutex> lock(mu);
    DeviceInfo &c = cache[dev];
    if (!c.ok) {
        if (cudaDeviceGetAttribute(&c.sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return LLOOM_ERR_DEVICE;
        if (cudaDeviceGetAttribute(&c.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
            return LLOOM_ERR_DEVICE;
        if (cudaDeviceGetAttribute(&c.smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess)
            return LLOOM_ERR_DEVICE;
        if (cudaDeviceGetAttribute(&c.smem_reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
            return LLOOM_ERR_DEVICE;
        if (cudaDeviceGetAttribute(&c.cc_major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) return LLOOM_ERR_DEVICE;
        if (c.cc_major != 10) return LLOOM_ERR_DEVICE;  // sm_100a code only
        c.ok = true;
    }
    out = c;
    return LLOOM_OK;
}

static int64_t weight_row_bytes(int dtype, int64_t k) {
    return k / lloom_b200_block_elems(dtype) * lloom_b200_block_bytes(dtype);
}

constexpr int64_t kMaxGridY = 65535;

// ---- GEMV launch planning ----

static cudaError_t launch_gemv_dp4a(const GemvParams &p, dim3 grid, int smem, bool overlap, int rw, cudaStream_t stream) {
    switch (p.w_dtype) {
    case LLOOM_Q8_0: return launch_gemv_dp4a_q8_0(p, grid, smem, overlap, rw, stream);
    case LLOOM_Q4_K: return launch_gemv_dp4a_q4k(p, grid, smem, overlap, rw, stream);
    case LLOOM_Q6_K: return launch_gemv_dp4a_q6k(p, grid, smem, overlap, rw, stream);
    case LLOOM_Q5_K: return launch_gemv_dp4a_q5k(p, grid, smem, overlap, rw, stream);
    case LLOOM_Q4_0: return launch_gemv_dp4a_q4_0(p, grid, smem, overlap, rw, stream);
    case LLOOM_Q5_0: return launch_gemv_dp4a_q5_0(p, grid, smem, overlap, rw, stream);
    }
    return cudaErrorInvalidValue;
}

static cudaError_t launch_mma(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream) {
    switch (p.w_dtype) {
    case LLOOM_Q8_0: return launch_mma_q8_0(p, map, nt, grid_x, grid_y, smem, overlap, stream);
    case LLOOM_Q4_K: return launch_mma_q4k(p, map, nt, grid_x, grid_y, smem, overlap, stream);
    case LLOOM_Q6_K: return launch_mma_q6k(p, map, nt, grid_x, grid_y, smem, overlap, stream);
    case LLOOM_Q5_K: return launch_mma_q5k(p, map, nt, grid_x, grid_y, smem, overlap, stream);
    case LLOOM_Q4_0: return launch_mma_q4_0(p, map, nt, grid_x, grid_y, smem, overlap, stream);
    case LLOOM_Q5_0: return launch_mma_q5_0(p, map, nt, grid_x, grid_y, smem, overlap, stream);
    }
    return cudaErrorInvalidValue;
}

// ---- tensor-core skinny product: planning ----

// How the m activation rows are laid out, a function of m and the format alone (the activation image is made before a matrix is
// known and serves a group of them): tiles of eight rows, in groups of at most six -- a CTA works on one group -- of equal size.
// A group of five is padded to six where its two column parts, which would share the middle tile, run better apart: Q4_K
// [14336, 4096] 37 rows 34.8 -> 33.0 us, 80 rows 58.4 -> 54.5, 112 rows 81.2 -> 75.3, Q4_0 108.5 -> 105.9, Q5_K level or 1 to 3 % better;
// Q6_K, Q8_0 and Q5_0 lose 1 to 4 %.
constexpr int64_t kMmaGroupTiles = 6;
struct MmaActs {
    int tiles = 0, group_nt = 0, groups = 0;
};
static MmaActs mma_acts(int w_dtype, int64_t m) {
    MmaActs a;
    const int64_t nt = (m + 7) / 8;
    a.groups = (int)((nt + kMmaGroupTiles - 1) / kMmaGroupTiles);
    a.group_nt = (int)((nt + a.groups - 1) / a.groups);
    if (a.group_nt == 5 && (w_dtype == LLOOM_Q4_K || w_dtype == LLOOM_Q5_K || w_dtype == LLOOM_Q4_0)) a.group_nt = 6;
    a.tiles = a.groups * a.group_nt;
    return a;
}
static int64_t mma_image_bytes(int w_dtype, int64_t m, int64_t k) {
    return (int64_t)mma_acts(w_dtype, m).tiles * ((k + 255) / 256) * image_unit_bytes(w_dtype, image_rows(m));
}

// Whether the kernel quantizes the activations itself (as its prologue, every CTA all rows): up to 64 256-element blocks,
// four per warp.  Measured per call at k = 4096, prologue against quantizer kernel: Q8_0 [4096, 4096], 3 / 4 rows alone 18.8 / 19.4
// against 20.7 / 20.8 us; Q4_K [14336, 4096] 22.9 / 23.6 against 24.1 / 24.1; eight rows are level or behind.  In a chain of
// launches (a caller who has asked for them to overlap) the quantizer kernel runs beside the product in front, where the prologue's
// time is all the forward's own: up to 32 blocks then ([4096, 4096] Q4_K / Q8_0, 4 rows, graph of launches: 7.0 / 7.7 against
// 5.4 / 7.1 us; [8192, 2048] Q6_K / Q8_0, 4 rows: 7.3 / 7.1 against 7.5 / 8.1).
static bool mma_fused(int64_t m, int64_t k) { return m <= 8 && m * ((k + 255) / 256) <= (launch_overlap() > 0 ? 32 : 64); }

// One row of activations against long rows of weights: the tensor-core kernel (eight slots along a row, sixteen warps on a
// tile or two) instead of the dp4a kernel (a warp along a row): [4096, 14336] Q4_K 11.3 / 13.1 us, Q6_K 15.3 / 16.9,
// Q8_0 17.0 / 19.7; at k = 8192 they are level.  Rows that start anywhere reach the former by slower copies.
// In a chain of launches (a caller who has asked for them to overlap) the dp4a kernel's CTAs sit beside their neighbours, which
// one that fills an SM alone cannot: a decoder layer's seven matmuls, dp4a against tensor cores for its down projection, Q4_K 43.7 /
// 46.7 us, Q6_K 63.6 / 67.6 (grouped 55.8 / 63.9); Q8_0 65.2 / 64.7, so the 32-element formats keep the latter.  (A chain of nothing
// but down projections: Q4_K 13.1 / 9.8, Q8_0 20.1 / 15.0.)
static bool long_rows(int w_dtype, int64_t k) {
    return k > 10240 && weight_row_bytes(w_dtype, k) % 16 == 0 && (act_is_q8_0(w_dtype) || launch_overlap() <= 0);
}

enum MmaActSource { kActImage, kActValues, kActBlocks };  // image in global memory; quantized / rearranged in the prologue

struct MmaPlan {
    bool ok = false;
    int nt = 0, tn = 0, split = 0, tr = 0, grid_x = 0, grid_y = 0, stages = 0, slice_sb = 0, boxes = 0;
    bool stream = false;
    bool two = false;  // two sums per warp
    int64_t pitch = 0, act_off = 0, stage = 0, red = 0, resident = 0;
};

// Up to eight rows of Q4_K / Q5_K against three or more weight tiles per CTA: four warps on a tile, each with the sums of two
// slots, instead of eight with one -- four tiles at a time, half the warps meeting in shared memory, the same bits.  Graph of
// launches, with / without, 8 rows: [14336, 4096] Q4_K 11.8 / 12.4 us, Q5_K 13.9 / 14.6, [8192, 2048] 5.3 / 6.0, 5.7 / 6.6; a layer
// with SiLU and product on the stores, 2 rows of Q4_K, 53.3 / 57.5.  With two tiles per CTA eight warps are level or better
// ([4096, 14336] 10.5 / 11.0); Q6_K and Q8_0 lose ([14336, 4096] 17.4 / 16.9, 18.7 / 18.5).
static bool two_sums(int w_dtype, int64_t tiles_per_cta) {
    return (w_dtype == LLOOM_Q4_K || w_dtype == LLOOM_Q5_K) && tiles_per_cta >= 3;
}

// Warps of a CTA: TR row tiles x S slots x TN column parts, at most sixteen.  How an output's sum is split depends on
// m and k alone.  Up to sixteen activation rows: eight slots, so that a CTA with one or two tiles -- all there is of a
// matrix of a few thousand rows on 148 SMs -- keeps sixteen warps busy; more rows: four, each warp with more columns.
static MmaPlan mma_plan(const DeviceInfo &di, int w_dtype, int64_t m, int64_t n, int64_t k, MmaActSource source, int64_t out_bytes) {
    MmaPlan pl;
    const MmaActs acts = mma_acts(w_dtype, m);
    if (source != kActImage && m > 8) return pl;
    const int64_t nsb = (k + 255) / 256, unit = image_unit_bytes(w_dtype, image_rows(m));
    const int64_t sb_bytes = 256 / lloom_b200_block_elems(w_dtype) * lloom_b200_block_bytes(w_dtype);
    pl.grid_y = acts.groups;
    pl.tn = acts.group_nt > 3 ? 2 : 1;
    pl.nt = (acts.group_nt + pl.tn - 1) / pl.tn;
    pl.split = pl.nt <= 2 && pl.tn == 1 ? 8 : 4;
    while (pl.split > 1 && pl.split / 2 >= nsb) pl.split /= 2;
    const int64_t total = (n + kMmaTileRows - 1) / kMmaTileRows;
    const int64_t ctas = di.sm_count / pl.grid_y > 0 ? di.sm_count / pl.grid_y : 1;
    pl.grid_x = (int)(total < ctas ? total : ctas);
    const int64_t per_cta = (total + pl.grid_x - 1) / pl.grid_x;
    pl.two = pl.split == 8 && pl.nt == 1 && m > 1 && two_sums(w_dtype, per_cta) && weight_row_bytes(w_dtype, k) % 16 == 0;
    if (pl.two) pl.split = 4;
    // Fragment loads of eight rows hit distinct banks when rows are an odd multiple of 8 words apart (formats read two words
    // per lane) or of 4 words (one word per lane).
    const int bank_words = w_dtype == LLOOM_Q4_K || w_dtype == LLOOM_Q5_K || w_dtype == LLOOM_Q8_0 ? 8 : 4;
    if (weight_row_bytes(w_dtype, k) % 16 == 0) {  // tiled TMA: boxes of at most 256 eight-byte elements
        pl.slice_sb = pl.two ? 8 : pl.split;
        for (pl.boxes = 1;; pl.boxes *= 2) {
            const int64_t w = pl.slice_sb / pl.boxes * sb_bytes;
            pl.pitch = bank_pitch(w + (w % 16 != 0 || (pl.slice_sb * sb_bytes) % 16 != 0 ? 16 : 0), bank_words);
            if (pl.pitch <= 2048) break;
        }
    }
    // other row lengths: long slices, about 4 KB of a row per copy if stages of that length fit
    int64_t longest = pl.boxes ? 1 : 4096 / (pl.split * sb_bytes);
    if (longest > (nsb + pl.split - 1) / pl.split) longest = (nsb + pl.split - 1) / pl.split;
    if (longest < 1) longest = 1;
    int tr_max = kMmaWarps / (pl.split * pl.tn);
    if (tr_max > 4) tr_max = 4;
    if (tr_max * pl.tn > kMmaMaxTeams) tr_max = kMmaMaxTeams / pl.tn;
    const int64_t res = nsb * acts.group_nt * unit;
    for (int64_t q = longest; q >= 1; q = q > 1 ? q / 2 : 0)
    for (int limit = tr_max; limit >= 1; limit = q > 1 ? 0 : limit - 1) {
        if (!pl.boxes) {
            pl.slice_sb = (int)(pl.split * q);
            pl.pitch = bank_pitch((nsb < pl.slice_sb ? nsb : pl.slice_sb) * sb_bytes + 32, bank_words);
        }
        const int64_t rounds = (per_cta + limit - 1) / limit;
        pl.tr = (int)((per_cta + rounds - 1) / rounds);
        pl.red = pl.split > 1 ? (int64_t)pl.tr * pl.tn * (pl.split - 1) * pl.nt * 512 : 0;
        const int64_t wstage = (int64_t)pl.tr * kMmaTileRows * pl.pitch * (pl.boxes > 0 ? pl.boxes : 1);
        // (di.smem_reserved: what a CTA of the next forward's quantizer takes beside this one)
        const int64_t room = (int64_t)di.max_smem_optin - di.smem_reserved - kMmaBarBytes - pl.red - out_bytes - kMmaSlack;
        // resident activations where the prologue makes them, and where several tile groups would fetch them again
        pl.stream = false;
        pl.resident = (res + 127) / 128 * 128;
        pl.stage = wstage;
        pl.act_off = wstage;
        int64_t stages = (room - pl.resident) / wstage;
        if (source == kActImage && (pl.grid_y > 1 || rounds == 1 || stages < 2)) {
            pl.stream = true;
            pl.resident = 0;
            pl.stage = (wstage + pl.slice_sb * acts.group_nt * unit + 127) / 128 * 128;
            stages = room / pl.stage;
        }
        if (stages < 2) continue;
        pl.stages = (int)(stages < kMmaStages ? stages : kMmaStages);
        pl.ok = true;
        return pl;
    }
    return pl;
}

struct PeerFlags {  // one flag array per GPU: kMaxPeers slots written by the peers + this GPU's call counter
    unsigned int *f[kMaxPeers];
};

// Where the outputs go, beyond the plain y: the fused gather (output buffers of all GPUs, own included, already offset
// to this shard's column), a block on the store, and the flag traffic of a gather with its barrier folded in.
struct GemvOut {
    int n_peers = 0;
    float *y[kMaxPeers] = {};
    int store = LLOOM_STORE_PLAIN;
    int rank = 0;
    bool publish = false;
    unsigned int *flags[kMaxPeers] = {};
    const unsigned int *wait_flags = nullptr;
    int wait_peers = 0;
};

// Several matrices of one dtype and k behind one launch (the activations are shared).
struct GemvGroup {
    int count = 0;
    const uint8_t *w[kMaxGroup] = {};
    float *y[kMaxGroup] = {};
    int64_t n[kMaxGroup] = {};
    int64_t ldy[kMaxGroup] = {};
    int store[kMaxGroup] = {};
    const uint32_t *moe_ids = nullptr;  // routed experts: matrix g = expert moe_ids[g] of the stack at `w` of the launch
    int moe_experts = 0;
    int moe_id_words = 1;  // 32-bit words per id (2: 64-bit ids, the low word counts)
    int64_t items = 1;     // groups of the launch (blockIdx.y): item i has ids and outputs of its own, activation row (item0 + i) / x_per
    int64_t x_per = 1;
    int64_t item0 = 0;
};

// The C entries: f32 in and out, launch overlap as set by lloom_b200_set_launch_overlap.
static FwdIo default_io() {
    FwdIo io;
    io.overlap = launch_overlap() > 0;
    return io;
}
static bool elem_type_ok(int t) { return t == LLOOM_F32 || t == LLOOM_F16 || t == LLOOM_BF16; }

// What both decode kernels need to know of a launch.
static void fill_params(GemvParams &p, int w_dtype, const void *w, const void *act, const void *x, void *y, int64_t m, int64_t n,
                        int64_t k, int64_t ldy, const FwdIo &io, const GemvOut *out) {
    memset(&p, 0, sizeof(p));
    p.w = (const uint8_t *)w;
    p.act = (const uint8_t *)act;
    p.x = x;
    p.y = (float *)y;
    p.x_type = io.x_type;
    p.y_type = io.y_type;
    p.ldy = ldy;
    p.row_bytes = weight_row_bytes(w_dtype, k);
    p.w_bytes = n * p.row_bytes;
    p.n = (int)n;
    p.k = (int)k;
    p.m = (int)m;
    p.w_dtype = w_dtype;
    p.nchunks = 1;
    if (out) {
        p.n_peers = out->n_peers;
        p.store_mode = out->store;
        p.publish = out->publish ? 1 : 0;
        p.peer_rank = out->rank;
        p.wait_flags = out->wait_flags;
        p.wait_peers = out->wait_peers;
        for (int g = 0; g < out->n_peers; ++g) {
            p.y_peer[g] = out->y[g];
            p.peer_flags[g] = out->flags[g];
        }
    }
}

// Room to stage a CTA's output rows for a fused gather (so that they leave for the peers in whole lines), if small.
static int64_t staging_bytes(int n_peers, int64_t m, int64_t rows_per_cta, int &pitch) {
    if (n_peers == 0) return 0;
    pitch = (int)((rows_per_cta + 3) / 4 * 4);
    const int64_t bytes = m * pitch * 4;
    return bytes <= 32 * 1024 ? bytes : 0;
}

// TMA view of the packed rows: boxes of 16 rows x `width` bytes, what lies past the matrix reads as zero.  (The driver's
// encoder is host arithmetic, 40 ns a call, so nothing is cached.)
static bool encode_rows_map(CUtensorMap &map, const void *w, int64_t n, int64_t row_bytes, int64_t width) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess) fn = nullptr;
        return (Encode)fn;
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes / 8, (cuuint64_t)n}, stride[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)width / 8, (cuuint32_t)kMmaTileRows}, step[2] = {1, 1};
    return encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<void *>(w), dims, stride, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launches the tensor-core kernel.  `acts`: the activation image, the values (m * superblocks bounded by shared memory) or
// canonical blocks, as `source` says.  LLOOM_ERR_SHAPE: no plan (activations made in the prologue that do not fit).
static int mma_launch(int w_dtype, const void *w, MmaActSource source, const void *acts, void *y, int64_t m, int64_t n, int64_t k,
                      int64_t ldy, cudaStream_t stream, const FwdIo &io, const GemvOut *out = nullptr) {
    DeviceInfo di;
    int rc = device_info(di);
    if (rc != LLOOM_OK) return rc;
    GemvParams p;
    fill_params(p, w_dtype, w, source == kActBlocks ? acts : nullptr, source == kActValues ? acts : nullptr, y, m, n, k, ldy, io, out);
    const int64_t total = (n + kMmaTileRows - 1) / kMmaTileRows, grid = total < di.sm_count ? total : di.sm_count;
    int pitch = 0;
    int64_t out_bytes = (staging_bytes(p.n_peers, m, (total + grid - 1) / grid * kMmaTileRows, pitch) + 127) / 128 * 128;
    MmaPlan pl = mma_plan(di, w_dtype, m, n, k, source, out_bytes);
    if (!pl.ok && out_bytes > 0) pl = mma_plan(di, w_dtype, m, n, k, source, out_bytes = 0);
    if (!pl.ok) return LLOOM_ERR_SHAPE;
    p.img = source == kActImage ? (const uint8_t *)acts : nullptr;
    p.img_unit = image_unit_bytes(w_dtype, image_rows(m));
    p.group_nt = mma_acts(w_dtype, m).group_nt;
    p.nsb = (int)((k + 255) / 256);
    p.split = pl.split;
    p.col_parts = pl.tn;
    p.tile_rows_cta = pl.tr * kMmaTileRows;
    const int sb_bytes = (int)(256 / lloom_b200_block_elems(w_dtype) * lloom_b200_block_bytes(w_dtype));
    p.slice_sb = pl.slice_sb;
    p.slice_bytes = pl.slice_sb * sb_bytes;
    p.boxes = pl.boxes;
    p.box_sb = pl.boxes ? pl.slice_sb / pl.boxes : 0;
    p.box_step = p.box_sb * sb_bytes / 8;
    p.box_bytes = kMmaTileRows * (int)pl.pitch;
    p.row_pitch = (int)pl.pitch;
    p.second = !pl.two ? 0 : pl.boxes > 1 ? p.box_bytes : pl.split * sb_bytes;
    p.act_stream = pl.stream ? 1 : 0;
    p.act_stage_off = (int)pl.act_off;
    p.act_bytes = (int)pl.resident;
    p.act_copy = (int)((int64_t)p.nsb * p.group_nt * p.img_unit);
    p.red_bytes = (int)pl.red;
    p.out_bytes = (int)out_bytes;
    p.out_pitch = out_bytes > 0 ? pitch : 0;
    p.stages = pl.stages;
    p.stage_bytes = (int)pl.stage;
    p.n_cwarps = pl.tr * pl.tn * pl.split;
    const int smem = (int)(kMmaBarBytes + pl.red + pl.resident + out_bytes + pl.stages * pl.stage + kMmaSlack);
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    if (pl.boxes && !encode_rows_map(map, w, n, p.row_bytes, pl.pitch)) return LLOOM_ERR_DEVICE;
    return launch_status(launch_mma(p, map, pl.nt, pl.grid_x, pl.grid_y, smem, io.overlap, stream));
}

// Launches the dp4a GEMV (one activation row; two for a group of matrices).  Exactly one of `act` (canonical activation blocks) and `x`
// (activations of type io.x_type, quantized in the kernel's prologue) is non-null.  With a group, w / y / n / ldy are
// ignored (n = total rows).
static int gemv_launch(int w_dtype, const void *w, const void *act, const void *x, void *y, int64_t m, int64_t n,
                       int64_t k, int64_t ldy, cudaStream_t stream, const FwdIo &io, const GemvOut *out = nullptr,
                       const GemvGroup *group = nullptr) {
    DeviceInfo di;
    int rc = device_info(di);
    if (rc != LLOOM_OK) return rc;
    GemvParams p;
    fill_params(p, w_dtype, w, act, x, y, m, n, k, ldy, io, out);
    p.act_bytes = (int)act_plane_bytes(w_dtype, m, k);
    p.unit_bytes = (int)((act_is_q8_0(w_dtype) ? 2 : 1) * lloom_b200_block_bytes(w_dtype));
    int items = 1;
    if (group) {
        p.n_group = group->count;
        int64_t off = 0;
        for (int g = 0; g < group->count; ++g) {
            p.gw[g] = group->w[g];
            p.gy[g] = group->y[g];
            p.gldy[g] = group->ldy[g];
            p.gstore[g] = group->store[g];
            p.goff[g] = (int)off;
            off += group->n[g];
        }
        p.goff[group->count] = (int)off;
        p.n = (int)off;
        n = off;
        p.moe_ids = group->moe_ids;
        p.moe_experts = group->moe_experts;
        p.moe_id_words = group->moe_id_words;
        p.x_per = (unsigned)group->x_per;
        p.item0 = (unsigned)group->item0;
        items = (int)group->items;
    }
    // lanes per row: one lane per unit (superblock, or pair of 32-element blocks), rounded up to a power of two
    const int64_t units = k / (act_is_q8_0(w_dtype) ? 64 : 256);
    int lpr_log2 = 0;
    while ((1 << lpr_log2) < units && lpr_log2 < 5) ++lpr_log2;
    p.lpr_log2 = lpr_log2;
    const int groups = 32 >> lpr_log2;
    // A stage holds one tile of rows, widened to 16-byte boundaries, plus slack for the word-wide
    // over-read of the unaligned loaders.
    const int64_t pad = (p.row_bytes % 16 == 0) ? 16 : 48;
    // one CTA per SM; several items share the SMs, two CTAs on each
    int grid = items == 1 ? di.sm_count : (2 * di.sm_count + items - 1) / items;
    if ((int64_t)grid > n) grid = (int)n;
    // Tile shapes {consumer warps, rows per lane}; the first that leaves room for at least two stages wins.  Two rows per
    // lane share the activation loads; where the CTA's rows fill the tiles of one row per lane much better, those win
    // ([14336, 4096]: 97 rows per SM are 7 tiles of 16 or 4 of 32).  A grouped launch runs the eight-warp, one-row-per-lane
    // shapes only, side by side with its neighbour in the stream first (two CTAs per SM).  A single matrix gets a side-by-side
    // shape where the caller has asked for chains of launches to overlap (lloom_b200_set_launch_overlap): graph of launches,
    // with / without: Q4_K [4096, 4096] 4.0 / 4.4 us, [8192, 2048] 3.4 / 3.9, Q8_0 [14336, 4096] 14.0 / 14.9, [8192, 2048] 5.1 / 6.0; a
    // decoder layer's seven matmuls Q4_K 43.7 / 49.0, Q6_K 63.6 / 69.6; past 128 MB what a neighbour saves no longer counts (Q6_K
    // [128256, 4096] 75.3 / 69.8).  For calls launched one by one it does not pay: a decoder layer of
    // separate calls takes 50 us with it and 46 without.  A row's bits are the same in every shape.
    const bool chain = !group && io.overlap && launch_overlap() > 0 && n * p.row_bytes <= (128 << 20);
    struct Shape { int cw, rw; bool half; };
    Shape shapes[12];
    int ns = 0;
    if (group) {
        shapes[ns++] = {8, 1, true};
        shapes[ns++] = {8, 1, false};
    } else {
        const int64_t rows = (n + grid - 1) / grid, tile = 8 * groups;
        const int64_t fill1 = (rows + tile - 1) / tile * tile, fill2 = (rows + 2 * tile - 1) / (2 * tile) * (2 * tile);
        if (chain) {
            if (w_dtype == LLOOM_Q8_0) shapes[ns++] = {12, 1, true};
            for (int c : {8, 4, 2, 1}) shapes[ns++] = {c, 1, true};
        }
        if (fill1 < fill2 && (fill2 - rows) * 5 > rows) shapes[ns++] = {8, 1, false};
        const int full[5][2] = {{8, 2}, {8, 1}, {4, 1}, {2, 1}, {1, 1}};
        for (auto &f : full) shapes[ns++] = {f[0], f[1], false};
    }
    int out_pitch = 0;
    const int64_t out_want = staging_bytes(p.n_peers, m, (n + grid - 1) / grid, out_pitch);
    for (int si = 0; si < ns; ++si) {
        const int cw = shapes[si].cw, rw = shapes[si].rw;
        const int64_t per_block = shapes[si].half ? (int64_t)(di.smem_per_sm - 2 * di.smem_reserved) / 2 / 16 * 16
                                                  : (int64_t)di.max_smem_optin;
        int64_t budget = per_block - 128 - p.act_bytes;
        int64_t stage = round16((int64_t)cw * groups * rw * p.row_bytes + pad);
        p.nchunks = 1;
        p.chunk_units = 0;
        p.lpr_log2 = lpr_log2;
        if (budget < 2 * stage) {
            // Long rows in a side-by-side shape: cut the rows into pieces of 16 units (32 for 64-element units), so
            // that a stage is 16 (8) rows x one piece -- the tile the kernel streams at K = 4096 -- instead of giving
            // up the overlap between consecutive launches for a one-CTA-per-SM shape.
            if (!shapes[si].half || m != 1 || cw > 8 || p.row_bytes % 16 != 0) continue;
            const int cu = act_is_q8_0(w_dtype) ? 32 : 16, cl = act_is_q8_0(w_dtype) ? 5 : 4;
            if (units <= cu || ((int64_t)cu * p.unit_bytes) % 16 != 0) continue;
            const int64_t pstage = round16((int64_t)cw * (32 >> cl) * rw * cu * p.unit_bytes + pad);
            if (budget < 2 * pstage) continue;
            stage = pstage;
            p.nchunks = (int)((units + cu - 1) / cu);
            p.chunk_units = cu;
            p.lpr_log2 = cl;
        }
        p.out_bytes = 0;
        p.out_pitch = 0;
        if (out_want > 0 && budget - out_want >= 2 * stage) {
            p.out_bytes = (int)out_want;
            p.out_pitch = out_pitch;
            budget -= out_want;
        }
        int64_t stages = budget / stage;
        if (stages > kMaxStages) stages = kMaxStages;
        p.n_cwarps = cw;
        p.stages = (int)stages;
        p.stage_bytes = (int)stage;
        const int smem = 128 + p.act_bytes + p.out_bytes + (int)(stages * stage);
        return launch_status(launch_gemv_dp4a(p, dim3((unsigned)grid, (unsigned)items), smem, io.overlap, rw, stream));
    }
    return LLOOM_ERR_SHAPE;  // one row of weights plus the activations does not fit in shared memory
}

static int check_common(int w_dtype, int64_t m, int64_t n, int64_t k) {
    if (!supported_weight(w_dtype)) return LLOOM_ERR_DTYPE;
    if (m <= 0 || n <= 0 || k <= 0) return LLOOM_ERR_SHAPE;
    if (k % lloom_b200_block_elems(w_dtype) != 0) return LLOOM_ERR_SHAPE;
    if (k % 64 != 0) return LLOOM_ERR_SHAPE;  // kernels work on 64-element items
    if (m > (1 << 24) || n > (1 << 30) || k > (1 << 24)) return LLOOM_ERR_SHAPE;
    return LLOOM_OK;
}

static bool aligned(const void *p, uintptr_t a) { return ((uintptr_t)p & (a - 1)) == 0; }

// ---- built-in scratch of lloom_b200_qmatmul_fwd_static ----
// Lives in every device's copy of this module until the process exits.  In host code the name
// below is only a host-side stand-in for the symbol, never a device address: the address a kernel
// may use is the one cudaGetSymbolAddress returns, looked up once per device.
static __device__ __align__(256) uint8_t g_static_scratch[LLOOM_B200_STATIC_SCRATCH_BYTES];

static int static_scratch_ptr(void **out) {
    static std::mutex mu;
    static void *cache[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LLOOM_ERR_DEVICE;
    std::lock_guard<std::mutex> lock(mu);
    if (!cache[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);  // `dev` is current here
        if (e != cudaSuccess) return launch_status(e);
        if (!p) return LLOOM_ERR_DEVICE;
        cache[dev] = p;
    }
    *out = cache[dev];
    return LLOOM_OK;
}

// Whether the skinny kernel serves this product: decode batches, prompts up to the row count where the tcgen05 GEMMs'
// higher rate pays for expanding the weights, and shapes those have no kernel for.  A function of m and k alone (not of n):
// a row shard takes the kernel its matrix takes.
static bool mma_serves(int w_dtype, int64_t m, int64_t k) {
    return m <= 128 || !gemm_supported(w_dtype, m, k, 1 << 30);
}
// With the weights already expanded the GEMM takes over earlier: its time hardly depends on m up to 128 rows or, while its
// tiles fit the SMs at once, on n, where the skinny kernel's grows with both.  Skinny / GEMM with image, us: Q4_K [14336,
// 4096] 48 rows 34 / 33, 64 rows 41 / 34, 128 rows 76 / 35; [8192, 4096] 64 rows 26 / 26, 80 rows 36 / 27; [5120, 5120] 80 rows
// 32 / 29; [4096, 4096] 96 rows 21 / 24, 112 rows 31 / 24.  Q6_K [14336, 4096] 64 rows 59 / 47, 128 rows 100 / 48; [5120, 5120] 80
// rows 44 / 38; [4096, 4096] 96 rows 27 / 31, 112 rows 36 / 31; [2048, 2048] 112 rows 16 / 18.  The 32-element formats drain their
// accumulators eight times as often: Q8_0 [14336, 4096] 96 rows 72 / 69, 128 rows 100 / 69; [11008, 4096] 96 rows 58 / 66, 112 rows
// 80 / 66; [8192, 8192] 112 rows 110 / 124.  (Without an image the GEMM of a narrow matrix would lose up to half, and a rule by
// n would give row shards other bits than their matrix.)
static bool image_pays(int w_dtype, int64_t m, int64_t n, int64_t k) {
    if (k < 2048) return false;  // the GEMM's set-up is most of a call then, and all of the above was measured from there on
    if (act_is_q8_0(w_dtype)) return m > 96 && n >= 10240;
    return (m > 96 && n >= 3072) || (m > 64 && n >= 5120) || (m > 48 && n >= 12288);
}
static bool mma_runs(int w_dtype, int64_t m, int64_t n, int64_t k, bool have_image) {
    return mma_serves(w_dtype, m, k) && !(have_image && image_pays(w_dtype, m, n, k) && gemm_supported(w_dtype, m, k, 1 << 30));
}
// Scratch of a product: the activation image of the skinny kernel, or the GEMM's images.
static int64_t product_scratch_bytes(int w_dtype, int64_t m, int64_t n, int64_t k, bool have_image) {
    if (mma_runs(w_dtype, m, n, k, have_image)) return (mma_image_bytes(w_dtype, m, k) + 255) / 256 * 256;
    return gemm_scratch_bytes(w_dtype, m, n, k, have_image);
}

// Activations to the image (`scratch`), then the product, for any m.
static int mma_forward(int w_dtype, const void *w_blocks, const void *act, const void *x, void *y, int64_t m, int64_t n, int64_t k,
                       int64_t ldy, void *scratch, cudaStream_t stream, const FwdIo &io, const GemvOut *out = nullptr) {
    constexpr int64_t kRows = kMaxGridY * kMmaGroupTiles * 8;  // of one launch: a group of activation tiles per blockIdx.y
    for (int64_t r = 0; r < m; r += kRows) {
        const int64_t rows = m - r < kRows ? m - r : kRows;
        const MmaActs acts = mma_acts(w_dtype, rows);
        int rc = launch_status(
            act ? launch_blocks_image(w_dtype, (const uint8_t *)act + r * lloom_b200_act_row_bytes(w_dtype, k), (uint8_t *)scratch, rows, k,
                                      acts.group_nt, stream)
                : launch_quantize_image(w_dtype, (const uint8_t *)x + r * k * elem_bytes(io.x_type), io.x_type, (uint8_t *)scratch, rows, k,
                                        acts.tiles, acts.group_nt, io.overlap, stream));
        if (rc != LLOOM_OK) return rc;
        rc = mma_launch(w_dtype, w_blocks, kActImage, scratch, (uint8_t *)y + r * ldy * elem_bytes(io.y_type), rows, n, k, ldy, stream, io, out);
        if (rc != LLOOM_OK) return rc;
    }
    return LLOOM_OK;
}

// Decode forward (m <= 8) after argument checks: outputs to `y` or to the peers' buffers.  One row: dp4a kernel with the
// quantizer as its prologue.  More: the tensor-core kernel, quantizer in its prologue for short batches, else a launch of
// its own.
static int decode_fwd(int w_dtype, const void *w_blocks, const void *x, void *y, int64_t m, int64_t n, int64_t k,
                      int64_t ldy, void *scratch, void *stream, const FwdIo &io, const GemvOut *out) {
    int rc;
    // activations that an earlier fused gather delivers may only be read by the kernel that waits for that gather
    const bool must_fuse = out && out->wait_flags;
    if (m == 1 && !long_rows(w_dtype, k)) {
        rc = gemv_launch(w_dtype, w_blocks, nullptr, x, y, m, n, k, ldy, (cudaStream_t)stream, io, out);
        if (rc != LLOOM_ERR_SHAPE) return rc;  // else: a row of weights does not fit its stages
    }
    if (must_fuse || mma_fused(m, k)) {
        rc = mma_launch(w_dtype, w_blocks, kActValues, x, y, m, n, k, ldy, (cudaStream_t)stream, io, out);
        if (rc != LLOOM_ERR_SHAPE) return rc;
        if (must_fuse) {  // rows too long to keep the batch in shared memory: row by row, the last one publishing
            for (int64_t r = 0; r < m; ++r) {
                GemvOut o = *out;
                for (int g = 0; g < o.n_peers; ++g) o.y[g] += r * ldy;
                if (r + 1 < m) o.publish = false;
                rc = gemv_launch(w_dtype, w_blocks, nullptr, (const uint8_t *)x + r * k * elem_bytes(io.x_type),
                                 (uint8_t *)y + r * ldy * elem_bytes(io.y_type), 1, n, k, ldy, (cudaStream_t)stream, io, &o);
                if (rc != LLOOM_OK) return rc;
            }
            return LLOOM_OK;
        }
    }
    return mma_forward(w_dtype, w_blocks, nullptr, x, y, m, n, k, ldy, scratch, (cudaStream_t)stream, io, out);
}

// Product of up to eight canonical activation rows, without scratch.
static int blocks_gemv(int w_dtype, const void *w_blocks, const void *act, void *y, int64_t m, int64_t n, int64_t k, int64_t ldy,
                       void *stream, const FwdIo &io) {
    int rc = LLOOM_ERR_SHAPE;
    if (m > 1) rc = mma_launch(w_dtype, w_blocks, kActBlocks, act, y, m, n, k, ldy, (cudaStream_t)stream, io);
    if (rc != LLOOM_ERR_SHAPE) return rc;
    const int64_t arow = lloom_b200_act_row_bytes(w_dtype, k);
    for (int64_t r = 0; r < m; ++r) {
        rc = gemv_launch(w_dtype, w_blocks, (const uint8_t *)act + r * arow, nullptr, (uint8_t *)y + r * ldy * elem_bytes(io.y_type), 1, n, k,
                         ldy, (cudaStream_t)stream, io);
        if (rc != LLOOM_OK) return rc;
    }
    return LLOOM_OK;
}

// Prefill product (m > 8) after argument checks.  Activations: canonical blocks in `act`, or values in `x` (every kernel
// quantizes them in the pass that lays them out).
static int gemm_dispatch(int w_dtype, const void *w_blocks, const void *w_image, const void *act, const void *x,
                         void *y, int64_t m, int64_t n, int64_t k, int64_t ldy, void *scratch, void *stream, const FwdIo &io) {
    if (mma_runs(w_dtype, m, n, k, w_image != nullptr))
        return mma_forward(w_dtype, w_blocks, act, x, y, m, n, k, ldy, scratch, (cudaStream_t)stream, io);
    return launch_status(gemm_forward(w_dtype, w_blocks, w_image, act, x, io.x_type, y, io.y_type, m, n, k, ldy, scratch,
                                      (cudaStream_t)stream));
}

static int fwd_checks(int w_dtype, const void *w_blocks, const void *x, const void *y, int64_t m, int64_t n, int64_t k,
                      int64_t ldy, const void *workspace, int64_t workspace_bytes, int64_t need) {
    int rc = check_common(w_dtype, m, n, k);
    if (rc != LLOOM_OK) return rc;
    if (ldy < n) return LLOOM_ERR_SHAPE;
    if (!w_blocks || !x || !y) return LLOOM_ERR_NULL;
    if (!workspace || workspace_bytes < need) return LLOOM_ERR_WORKSPACE;
    if (!aligned(workspace, 256) || !aligned(w_blocks, 16) || !aligned(x, 16) || !aligned(y, 4)) return LLOOM_ERR_ALIGN;
    return LLOOM_OK;
}

int qmatmul_forward(int w_dtype, const void *w_blocks, const void *w_image, const void *x, void *y, int64_t m, int64_t n, int64_t k,
                    int64_t ldy, int store, void *workspace, int64_t workspace_bytes, void *stream, const FwdIo &io) {
    const int64_t need = w_image ? lloom_b200_workspace_bytes_with_image(w_dtype, m, n, k) : lloom_b200_workspace_bytes(w_dtype, m, n, k);
    int rc = fwd_checks(w_dtype, w_blocks, x, y, m, n, k, ldy, workspace, workspace_bytes, need);
    if (rc != LLOOM_OK) return rc;
    if (!elem_type_ok(io.x_type) || !elem_type_ok(io.y_type)) return LLOOM_ERR_DTYPE;
    if (w_image && !aligned(w_image, 1024)) return LLOOM_ERR_ALIGN;
    if (store < LLOOM_STORE_PLAIN || store > LLOOM_STORE_MUL_INTO) return LLOOM_ERR_SHAPE;
    if (store != LLOOM_STORE_PLAIN && (m > 8 || io.y_type != LLOOM_F32)) return LLOOM_ERR_SHAPE;
    if (m <= 8) {
        GemvOut out;
        out.store = store;
        return decode_fwd(w_dtype, w_blocks, x, y, m, n, k, ldy, workspace, stream, io, store != LLOOM_STORE_PLAIN ? &out : nullptr);
    }
    if (w_image && lloom_b200_weight_image_bytes(w_dtype, n, k) <= 0) return LLOOM_ERR_SHAPE;  // no image exists for this shape
    return gemm_dispatch(w_dtype, w_blocks, w_image, nullptr, x, y, m, n, k, ldy, workspace, stream, io);
}

int qmatmul_forward_group(int w_dtype, int n_mats, const void *const *w_blocks, const void *x, float *const *ys, const int64_t *ns,
                          const int64_t *ldys, const int *stores, int64_t m, int64_t k, void *workspace, int64_t workspace_bytes,
                          void *stream, const FwdIo &io) {
    if (!elem_type_ok(io.x_type) || io.y_type != LLOOM_F32) return LLOOM_ERR_DTYPE;
    if (n_mats < 1 || n_mats > kMaxGroup) return LLOOM_ERR_SHAPE;
    if (!w_blocks || !x || !ys || !ns || !ldys) return LLOOM_ERR_NULL;
    if (m > 8) return LLOOM_ERR_SHAPE;
    GemvGroup group;
    group.count = n_mats;
    int64_t n_max = 0, n_total = 0;
    for (int g = 0; g < n_mats; ++g) {
        int rc = check_common(w_dtype, m, ns[g], k);
        if (rc != LLOOM_OK) return rc;
        if (ldys[g] < ns[g]) return LLOOM_ERR_SHAPE;
        if (!w_blocks[g] || !ys[g]) return LLOOM_ERR_NULL;
        if (!aligned(w_blocks[g], 16) || !aligned(ys[g], 4)) return LLOOM_ERR_ALIGN;
        const int store = stores ? stores[g] : LLOOM_STORE_PLAIN;
        if (store < LLOOM_STORE_PLAIN || store > LLOOM_STORE_MUL_INTO) return LLOOM_ERR_SHAPE;
        group.w[g] = (const uint8_t *)w_blocks[g];
        group.y[g] = ys[g];
        group.n[g] = ns[g];
        group.ldy[g] = ldys[g];
        group.store[g] = store;
        if (ns[g] > n_max) n_max = ns[g];
        n_total += ns[g];
    }
    if (n_total > (1ll << 30)) return LLOOM_ERR_SHAPE;
    const int64_t need = lloom_b200_workspace_bytes(w_dtype, m, n_max, k);
    if (!workspace || workspace_bytes < need) return LLOOM_ERR_WORKSPACE;
    if (!aligned(workspace, 256) || !aligned(x, 16)) return LLOOM_ERR_ALIGN;
    int rc;
    // One launch of the dp4a kernel for the whole group: one row, where it is the decode path anyway, and two rows of up to
    // 40 MB, where it spares a quantizer and a launch per matrix (graph, Q4_K / Q8_0: q|k|v of a 4096-wide model 11.5 -> 7.9, 14.3 ->
    // 10.3 us, two of [8192, 2048] 10.0 -> 7.4, 14.4 -> 12.0).  Larger groups gain little or nothing alone (two of [14336, 4096]
    // 21.5 -> 21.2, 34.3 -> 31.4; Q4_0 26.4 -> 28.3) and lose in a layer, whose next launches cannot start beside them (Q4_K
    // layer with groups 49.3 -> 55.8, Q8_0 70.5 -> 73.0).
    if (n_mats > 1 && (m == 1 || (m == 2 && n_total * weight_row_bytes(w_dtype, k) <= (40 << 20)))) {
        rc = gemv_launch(w_dtype, nullptr, nullptr, x, nullptr, m, 0, k, 0, (cudaStream_t)stream, io, nullptr, &group);
        if (rc != LLOOM_ERR_SHAPE) return rc;
    }
    // Otherwise the activations are quantized once and every matrix gets its own launch.
    uint8_t *scratch = (uint8_t *)workspace;
    if (m > 1) {
        const MmaActs acts = mma_acts(w_dtype, m);
        rc = launch_status(launch_quantize_image(w_dtype, x, io.x_type, scratch, m, k, acts.tiles, acts.group_nt, io.overlap,
                                                 (cudaStream_t)stream));
        if (rc != LLOOM_OK) return rc;
    }
    for (int g = 0; g < n_mats; ++g) {
        GemvOut out;
        out.store = group.store[g];
        rc = m > 1 ? mma_launch(w_dtype, group.w[g], kActImage, scratch, group.y[g], m, group.n[g], k, group.ldy[g], (cudaStream_t)stream, io, &out)
                   : decode_fwd(w_dtype, group.w[g], x, group.y[g], m, group.n[g], k, group.ldy[g], scratch, stream, io, &out);
        if (rc != LLOOM_OK) return rc;
    }
    return LLOOM_OK;
}

int indexed_moe_forward(int w_dtype, const void *w_experts, int64_t n_experts, int64_t n, int64_t k, const float *x, int64_t batch,
                        int64_t in_dim1, const void *ids, bool ids64, int64_t topk, float *out, void *workspace,
                        int64_t workspace_bytes, void *stream, const FwdIo &io) {
    int rc = check_common(w_dtype, 1, n, k);
    if (rc != LLOOM_OK) return rc;
    if (n_experts <= 0 || n_experts > (1 << 20) || batch <= 0 || topk <= 0 || topk > 0x7fffffff || (in_dim1 != 1 && in_dim1 != topk))
        return LLOOM_ERR_SHAPE;
    if (!w_experts || !x || !ids || !out) return LLOOM_ERR_NULL;
    if (n_experts * n > (1ll << 30)) return LLOOM_ERR_SHAPE;
    if (!aligned(w_experts, 16) || !aligned(x, 16) || !aligned(ids, ids64 ? 8 : 4) || !aligned(out, 4)) return LLOOM_ERR_ALIGN;
    const int64_t need = lloom_b200_workspace_bytes(w_dtype, 1, n, k);
    if (!workspace || workspace_bytes < need) return LLOOM_ERR_WORKSPACE;
    if (!aligned(workspace, 256)) return LLOOM_ERR_ALIGN;
    // One launch for all products: CTAs (x, y), y = a token with its experts as a group, or one product where the
    // activations (or the group size) are not shared.
    const bool share_x = in_dim1 == 1 && topk <= kMaxGroup;
    const int64_t items = share_x ? batch : batch * topk;
    GemvGroup group;
    group.count = share_x ? (int)topk : 1;
    for (int g = 0; g < group.count; ++g) {
        group.w[g] = (const uint8_t *)w_experts;  // replaced on the device by the routed expert
        group.y[g] = out + g * n;
        group.n[g] = n;
        group.ldy[g] = n;
        group.store[g] = LLOOM_STORE_PLAIN;
    }
    group.moe_ids = (const uint32_t *)ids;
    group.moe_experts = (int)n_experts;
    group.moe_id_words = ids64 ? 2 : 1;
    group.x_per = in_dim1 == 1 ? items / batch : 1;
    for (int64_t i0 = 0; i0 < items; i0 += kMaxGridY) {  // a launch may start in the middle of a token
        GemvGroup part = group;
        part.items = items - i0 < kMaxGridY ? items - i0 : kMaxGridY;
        part.item0 = i0 % group.x_per;
        part.moe_ids += i0 * group.count * group.moe_id_words;
        for (int g = 0; g < group.count; ++g) part.y[g] += i0 * group.count * n;
        rc = gemv_launch(w_dtype, w_experts, nullptr, x + i0 / group.x_per * k, nullptr, 1, 0, k, 0, (cudaStream_t)stream, io, nullptr, &part);
        if (rc != LLOOM_OK) return rc;
    }
    return LLOOM_OK;
}

int get_rows(int dtype, const void *blocks, int64_t rows, int64_t hidden, const void *ids, bool ids64, int64_t n_ids, float *out,
             void *stream, bool overlap) {
    if (!supported_weight(dtype)) return LLOOM_ERR_DTYPE;
    if (rows <= 0 || hidden <= 0 || n_ids <= 0 || hidden % lloom_b200_block_elems(dtype) != 0) return LLOOM_ERR_SHAPE;
    if (!blocks || !ids || !out) return LLOOM_ERR_NULL;
    if (!aligned(blocks, 16) || !aligned(out, 16) || !aligned(ids, ids64 ? 8 : 4)) return LLOOM_ERR_ALIGN;
    const int64_t per_row = hidden / 8;
    const unsigned threads = (unsigned)(per_row >= 256 ? 256 : (per_row + 31) / 32 * 32);
    if (n_ids > 0x7fffffff || ceil_div64(per_row, threads) > 65535) return LLOOM_ERR_SHAPE;
    const dim3 grid((unsigned)n_ids, (unsigned)ceil_div64(per_row, threads));
    cudaError_t e = cudaErrorInvalidValue;
    with_format(dtype, [&](auto fmt) {
        e = launch_early(get_rows_kernel<decltype(fmt)::value>, grid, threads, 0, overlap, (cudaStream_t)stream, (const uint8_t *)blocks, rows,
                         hidden, weight_row_bytes(dtype, hidden), (const uint32_t *)ids, ids64 ? 2 : 1, out);
    });
    return launch_status(e);
}

}  // namespace lloom

using namespace lloom;

extern "C" {

int lloom_b200_version(void) { return LLOOM_B200_VERSION; }

const char *lloom_b200_error_string(int status) {
    switch (status) {
    case LLOOM_OK: return "ok";
    case LLOOM_ERR_DTYPE: return "unsupported GgmlDType (weights: Q4_0, Q5_0, Q8_0, Q4_K, Q5_K, Q6_K)";
    case LLOOM_ERR_SHAPE: return "bad shape";
    case LLOOM_ERR_ALIGN: return "misaligned pointer";
    case LLOOM_ERR_NULL: return "null pointer";
    case LLOOM_ERR_WORKSPACE: return "workspace missing or too small";
    case LLOOM_ERR_LAUNCH: return "CUDA launch error";
    case LLOOM_ERR_TIMEOUT: return "device-side wait timed out";
    case LLOOM_ERR_DEVICE: return "not an sm_100 device";
    case LLOOM_ERR_STATIC_LIMIT: return "request exceeds the built-in scratch (m <= 8 and m * act_row_bytes <= 256 KiB)";
    }
    return "unknown status";
}

int lloom_b200_last_cuda_error(void) { return t_last_cuda_error; }

int lloom_b200_set_launch_overlap(int enable) {
    return g_launch_overlap.exchange(enable > 0 ? 1 : enable < 0 ? -1 : 0, std::memory_order_relaxed);
}

int lloom_b200_device_status(int *status_out) {
    if (!status_out) return LLOOM_ERR_NULL;
    TuRegistry &r = tu_registry();
    std::lock_guard<std::mutex> lock(r.mu);  // one reader at a time: the fetch goes through a per-unit landing word
    int status = 0;
    for (const TuHooks &h : r.hooks) {
        int v = 0;
        const cudaError_t e = h.fetch_status(&v, nullptr);  // device-side atomic exchange, then a synchronous read
        if (e != cudaSuccess) return launch_status(e);
        if (v != 0) status = v;
    }
    *status_out = status;
    return LLOOM_OK;
}

int lloom_b200_set_wait_limit_ns(uint64_t ns) {
    if (ns == 0) ns = kDefaultWaitNs;
    TuRegistry &r = tu_registry();
    std::lock_guard<std::mutex> lock(r.mu);
    for (const TuHooks &h : r.hooks) {
        const cudaError_t e = h.set_wait_limit((unsigned long long)ns);
        if (e != cudaSuccess) return launch_status(e);
    }
    return LLOOM_OK;
}

int64_t lloom_b200_block_elems(int dtype) {
    switch (dtype) {
    case LLOOM_Q8_0: case LLOOM_Q4_0: case LLOOM_Q5_0: return QK8_0;
    case LLOOM_Q4_K: case LLOOM_Q5_K: case LLOOM_Q6_K: case LLOOM_Q8_K: return QK_K;
    }
    return 0;
}

int64_t lloom_b200_block_bytes(int dtype) {
    switch (dtype) {
    case LLOOM_Q8_0: return Q8_0_BYTES;
    case LLOOM_Q4_K: return Q4K_BYTES;
    case LLOOM_Q6_K: return Q6K_BYTES;
    case LLOOM_Q8_K: return Q8K_BYTES;
    case LLOOM_Q4_0: return Q4_0_BYTES;
    case LLOOM_Q5_0: return Q5_0_BYTES;
    case LLOOM_Q5_K: return Q5K_BYTES;
    }
    return 0;
}

int lloom_b200_act_dtype(int w_dtype) {
    switch (w_dtype) {
    case LLOOM_Q8_0: case LLOOM_Q4_0: case LLOOM_Q5_0: return LLOOM_Q8_0;
    case LLOOM_Q4_K: case LLOOM_Q5_K: case LLOOM_Q6_K: return LLOOM_Q8_K;
    }
    return 0;
}

int64_t lloom_b200_act_row_bytes(int w_dtype, int64_t k) {
    const int adt = lloom_b200_act_dtype(w_dtype);
    if (!adt || k <= 0 || k % lloom_b200_block_elems(adt) != 0) return 0;
    return k / lloom_b200_block_elems(adt) * lloom_b200_block_bytes(adt);
}

int64_t lloom_b200_workspace_bytes(int w_dtype, int64_t m, int64_t n, int64_t k) {
    if (check_common(w_dtype, m, n, k) != LLOOM_OK) return 0;
    return product_scratch_bytes(w_dtype, m, n, k, false);
}

int64_t lloom_b200_workspace_bytes_with_image(int w_dtype, int64_t m, int64_t n, int64_t k) {
    if (check_common(w_dtype, m, n, k) != LLOOM_OK) return 0;
    return product_scratch_bytes(w_dtype, m, n, k, true);
}

int64_t lloom_b200_weight_image_bytes(int w_dtype, int64_t n, int64_t k) {
    if (check_common(w_dtype, 1, n, k) != LLOOM_OK) return 0;
    if (!gemm_supported(w_dtype, 9, k, 1 << 30)) return 0;
    return gemm_weight_image_bytes(w_dtype, n, k);
}

int lloom_b200_weight_image_build(int w_dtype, const void *w_blocks, int64_t n, int64_t k, void *image, int64_t image_bytes,
                                  void *stream) {
    int rc = check_common(w_dtype, 1, n, k);
    if (rc != LLOOM_OK) return rc;
    const int64_t need = lloom_b200_weight_image_bytes(w_dtype, n, k);
    if (need <= 0) return LLOOM_ERR_SHAPE;
    if (!w_blocks || !image) return LLOOM_ERR_NULL;
    if (image_bytes < need) return LLOOM_ERR_WORKSPACE;
    if (!aligned(w_blocks, 16) || !aligned(image, 1024)) return LLOOM_ERR_ALIGN;
    return launch_status(gemm_weight_image_build(w_dtype, w_blocks, n, k, image, (cudaStream_t)stream));
}

int lloom_b200_quantize_act(int w_dtype, const float *x, int64_t m, int64_t k, void *act_blocks, void *stream) {
    int rc = check_common(w_dtype, m, 1, k);
    if (rc != LLOOM_OK) return rc;
    if (!x || !act_blocks) return LLOOM_ERR_NULL;
    if (!aligned(x, 16) || !aligned(act_blocks, 4)) return LLOOM_ERR_ALIGN;
    return launch_status(launch_quantize_act(w_dtype, x, LLOOM_F32, m, k, act_blocks, default_io().overlap, (cudaStream_t)stream));
}

int lloom_b200_gemv(int w_dtype, const void *w_blocks, const void *act_blocks, float *y, int64_t m, int64_t n,
                    int64_t k, int64_t ldy, void *stream) {
    int rc = check_common(w_dtype, m, n, k);
    if (rc != LLOOM_OK) return rc;
    if (m > 8 || ldy < n) return LLOOM_ERR_SHAPE;
    if (!w_blocks || !act_blocks || !y) return LLOOM_ERR_NULL;
    if (!aligned(w_blocks, 16) || !aligned(act_blocks, 4) || !aligned(y, 4)) return LLOOM_ERR_ALIGN;
    return blocks_gemv(w_dtype, w_blocks, act_blocks, y, m, n, k, ldy, stream, default_io());
}

int lloom_b200_gemm(int w_dtype, const void *w_blocks, const void *act_blocks, float *y, int64_t m, int64_t n,
                    int64_t k, int64_t ldy, void *workspace, int64_t workspace_bytes, void *stream) {
    int rc = check_common(w_dtype, m, n, k);
    if (rc != LLOOM_OK) return rc;
    if (ldy < n) return LLOOM_ERR_SHAPE;
    if (!w_blocks || !act_blocks || !y) return LLOOM_ERR_NULL;
    if (!aligned(w_blocks, 16) || !aligned(act_blocks, 4) || !aligned(y, 4)) return LLOOM_ERR_ALIGN;
    if (m <= 8) return blocks_gemv(w_dtype, w_blocks, act_blocks, y, m, n, k, ldy, stream, default_io());  // needs no workspace
    const int64_t need = product_scratch_bytes(w_dtype, m, n, k, false);
    if (need > 0 && (!workspace || workspace_bytes < need)) return LLOOM_ERR_WORKSPACE;
    if (need > 0 && !aligned(workspace, 256)) return LLOOM_ERR_ALIGN;
    return gemm_dispatch(w_dtype, w_blocks, nullptr, act_blocks, nullptr, y, m, n, k, ldy, workspace, stream, default_io());
}

int lloom_b200_qmatmul_fwd(int w_dtype, const void *w_blocks, const float *x, float *y, int64_t m, int64_t n,
                           int64_t k, int64_t ldy, void *workspace, int64_t workspace_bytes, void *stream) {
    return qmatmul_forward(w_dtype, w_blocks, nullptr, x, y, m, n, k, ldy, LLOOM_STORE_PLAIN, workspace, workspace_bytes, stream,
                           default_io());
}

int lloom_b200_qmatmul_fwd_image(int w_dtype, const void *w_blocks, const void *w_image, const float *x, float *y,
                                 int64_t m, int64_t n, int64_t k, int64_t ldy, void *workspace, int64_t workspace_bytes,
                                 void *stream) {
    return qmatmul_forward(w_dtype, w_blocks, w_image, x, y, m, n, k, ldy, LLOOM_STORE_PLAIN, workspace, workspace_bytes, stream,
                           default_io());
}

int lloom_b200_qmatmul_fwd_typed(int w_dtype, const void *w_blocks, const void *w_image, const void *x, int x_type, void *y,
                                 int y_type, int64_t m, int64_t n, int64_t k, int64_t ldy, void *workspace,
                                 int64_t workspace_bytes, void *stream) {
    FwdIo io = default_io();
    io.x_type = x_type;
    io.y_type = y_type;
    return qmatmul_forward(w_dtype, w_blocks, w_image, x, y, m, n, k, ldy, LLOOM_STORE_PLAIN, workspace, workspace_bytes, stream, io);
}

int lloom_b200_qmatmul_fwd_store(int w_dtype, const void *w_blocks, const float *x, float *y, int64_t m, int64_t n,
                                 int64_t k, int64_t ldy, int store, void *workspace, int64_t workspace_bytes,
                                 void *stream) {
    if (m > 8) {
        const int rc = fwd_checks(w_dtype, w_blocks, x, y, m, n, k, ldy, workspace, workspace_bytes,
                                  lloom_b200_workspace_bytes(w_dtype, m, n, k));
        return rc != LLOOM_OK ? rc : LLOOM_ERR_SHAPE;
    }
    return qmatmul_forward(w_dtype, w_blocks, nullptr, x, y, m, n, k, ldy, store, workspace, workspace_bytes, stream, default_io());
}

int lloom_b200_qmatmul_fwd_group(int w_dtype, int n_mats, const void *const *w_blocks, const float *x, float *const *ys,
                                 const int64_t *ns, const int64_t *ldys, const int *stores, int64_t m, int64_t k,
                                 void *workspace, int64_t workspace_bytes, void *stream) {
    return qmatmul_forward_group(w_dtype, n_mats, w_blocks, x, ys, ns, ldys, stores, m, k, workspace, workspace_bytes, stream,
                                 default_io());
}

int lloom_b200_indexed_moe_forward(int w_dtype, const void *w_experts, int64_t n_experts, int64_t n, int64_t k,
                                   const float *x, int64_t batch, int64_t in_dim1, const uint32_t *ids, int64_t topk,
                                   float *out, void *workspace, int64_t workspace_bytes, void *stream) {
    return indexed_moe_forward(w_dtype, w_experts, n_experts, n, k, x, batch, in_dim1, ids, false, topk, out, workspace,
                               workspace_bytes, stream, default_io());
}

static int gather_common(int w_dtype, const void *w_shard, const float *x, int64_t m, int64_t n_shard, int64_t k,
                         int64_t ldy, int64_t col0, float *const *y_peers, int n_peers, void *workspace,
                         int64_t workspace_bytes, void *stream, GemvOut &peers) {
    int rc = check_common(w_dtype, m, n_shard, k);
    if (rc != LLOOM_OK) return rc;
    if (m > 8 || n_peers < 1 || n_peers > kMaxPeers || col0 < 0 || ldy < col0 + n_shard) return LLOOM_ERR_SHAPE;
    if (!w_shard || !x || !y_peers) return LLOOM_ERR_NULL;
    const int64_t need = lloom_b200_workspace_bytes(w_dtype, m, n_shard, k);
    if (!workspace || workspace_bytes < need) return LLOOM_ERR_WORKSPACE;
    if (!aligned(workspace, 256) || !aligned(w_shard, 16) || !aligned(x, 16)) return LLOOM_ERR_ALIGN;
    peers.n_peers = n_peers;
    for (int g = 0; g < n_peers; ++g) {
        if (!y_peers[g]) return LLOOM_ERR_NULL;
        if (!aligned(y_peers[g], 4)) return LLOOM_ERR_ALIGN;
        peers.y[g] = y_peers[g] + col0;
    }
    return decode_fwd(w_dtype, w_shard, x, peers.y[0], m, n_shard, k, ldy, workspace, stream, default_io(), &peers);
}

int lloom_b200_qmatmul_fwd_gather(int w_dtype, const void *w_shard, const float *x, int64_t m, int64_t n_shard, int64_t k,
                                  int64_t ldy, int64_t col0, float *const *y_peers, int n_peers, void *workspace,
                                  int64_t workspace_bytes, void *stream) {
    GemvOut peers;
    return gather_common(w_dtype, w_shard, x, m, n_shard, k, ldy, col0, y_peers, n_peers, workspace, workspace_bytes, stream,
                         peers);
}

int lloom_b200_qmatmul_fwd_gather_sync(int w_dtype, const void *w_shard, const float *x, int64_t m, int64_t n_shard,
                                       int64_t k, int64_t ldy, int64_t col0, float *const *y_peers, int n_peers, int rank,
                                       unsigned int *const *flag_peers, const unsigned int *wait_flags, void *workspace,
                                       int64_t workspace_bytes, void *stream) {
    if (n_peers < 1 || n_peers > kMaxPeers || rank < 0 || rank >= n_peers) return LLOOM_ERR_SHAPE;
    if (!flag_peers) return LLOOM_ERR_NULL;
    if (wait_flags && m > 2) return LLOOM_ERR_SHAPE;  // the wait sits in the GEMV's own quantizer prologue (m <= 2)
    GemvOut peers;
    peers.publish = true;
    peers.rank = rank;
    for (int g = 0; g < n_peers; ++g) {
        if (!flag_peers[g]) return LLOOM_ERR_NULL;
        if (!aligned(flag_peers[g], 4)) return LLOOM_ERR_ALIGN;
        peers.flags[g] = flag_peers[g];
    }
    peers.wait_flags = wait_flags;
    peers.wait_peers = wait_flags ? n_peers : 0;
    return gather_common(w_dtype, w_shard, x, m, n_shard, k, ldy, col0, y_peers, n_peers, workspace, workspace_bytes, stream,
                         peers);
}

int lloom_b200_qmatmul_fwd_after_gather(int w_dtype, const void *w_blocks, const float *x, float *y, int64_t m, int64_t n,
                                        int64_t k, int64_t ldy, const unsigned int *wait_flags, int n_peers,
                                        void *workspace, int64_t workspace_bytes, void *stream) {
    const int64_t need = lloom_b200_workspace_bytes(w_dtype, m, n, k);
    int rc = fwd_checks(w_dtype, w_blocks, x, y, m, n, k, ldy, workspace, workspace_bytes, need);
    if (rc != LLOOM_OK) return rc;
    if (m > 2 || n_peers < 1 || n_peers > kMaxPeers) return LLOOM_ERR_SHAPE;  // served where the quantizer is the GEMV's prologue
    if (!wait_flags) return LLOOM_ERR_NULL;
    GemvOut out;
    out.wait_flags = wait_flags;
    out.wait_peers = n_peers;
    return decode_fwd(w_dtype, w_blocks, x, y, m, n, k, ldy, workspace, stream, default_io(), &out);
}

// Waits (bounded) until every slot of this GPU's flag array has reached the GPU's own call counter: the gathered
// rows of the last lloom_b200_qmatmul_fwd_gather_sync on this stream are complete.  One warp, lane g polls slot g.
__global__ void peer_wait_kernel(int n_peers, const unsigned int *flags) {
    // let the stream's next kernel become resident (a GEMV starts streaming its weights) while this one waits for
    // the GEMV before it and then for the peers; that kernel's own griddepcontrol.wait holds it until this one is done
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int g = threadIdx.x;
    if (g >= n_peers) return;
    unsigned int want;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(want) : "l"(flags + kMaxPeers) : "memory");
    unsigned long long t0 = 0;
    for (uint32_t i = 0; i < kMaxSpins; ++i) {
        unsigned int seen;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(flags + g) : "memory");
        if ((int)(seen - want) >= 0) return;
        if ((i & 63) == 63) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > wait_limit_ns()) break;
        }
        __nanosleep(100);
    }
    atomicExch(&g_device_status, LLOOM_ERR_TIMEOUT);
}

// Cross-GPU barrier after a fused gather: one small kernel per GPU.  Each GPU bumps its own epoch, publishes it in
// slot [rank] of every GPU's flag array (system-scope release: the gather's stores, finished with the previous
// kernel on this stream, are visible before it) and waits until all slots of its own array have reached the
// epoch.  The wait is bounded in time; on a time-out the status word is set and the kernel returns.
__global__ void peer_barrier_kernel(int rank, int n_peers, PeerFlags flags) {
    __shared__ unsigned int s_epoch;
    // launched with programmatic serialization when launch overlap is on: resident early, it waits here for the
    // GEMV before it (and that GEMV's peer stores) to finish; the kernel behind it may become resident meanwhile
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    unsigned int *mine = flags.f[rank];
    if (threadIdx.x == 0) {
        s_epoch = mine[kMaxPeers] + 1;  // slot kMaxPeers: this GPU's call counter
        mine[kMaxPeers] = s_epoch;
        __threadfence_system();
    }
    __syncthreads();
    const unsigned int epoch = s_epoch;
    const int g = threadIdx.x;
    if (g >= n_peers) return;
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flags.f[g] + rank), "r"(epoch) : "memory");
    unsigned long long t0 = 0;
    for (uint32_t i = 0; i < kMaxSpins; ++i) {
        unsigned int seen;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(mine + g) : "memory");
        if ((int)(seen - epoch) >= 0) return;
        if ((i & 63) == 63) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > wait_limit_ns()) break;
        }
        __nanosleep(100);
    }
    atomicExch(&g_device_status, LLOOM_ERR_TIMEOUT);
}

static cudaError_t launch_one_warp(void (*kern)(int, const unsigned int *), int a, const unsigned int *b, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = launch_overlap() > 0 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, a, b);
}

int lloom_b200_peer_wait(int n_peers, const unsigned int *flags_own, void *stream) {
    if (n_peers < 1 || n_peers > kMaxPeers) return LLOOM_ERR_SHAPE;
    if (!flags_own) return LLOOM_ERR_NULL;
    return launch_status(launch_one_warp(peer_wait_kernel, n_peers, flags_own, (cudaStream_t)stream));
}

int lloom_b200_peer_barrier(int rank, int n_peers, unsigned int *const *flag_peers, void *stream) {
    if (n_peers < 1 || n_peers > kMaxPeers || rank < 0 || rank >= n_peers) return LLOOM_ERR_SHAPE;
    if (!flag_peers) return LLOOM_ERR_NULL;
    PeerFlags flags;
    for (int g = 0; g < kMaxPeers; ++g) {
        flags.f[g] = g < n_peers ? flag_peers[g] : nullptr;
        if (g < n_peers && !flags.f[g]) return LLOOM_ERR_NULL;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(32);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = launch_overlap() > 0 ? 1 : 0;
    return launch_status(cudaLaunchKernelEx(&cfg, peer_barrier_kernel, rank, n_peers, flags));
}

// Set-up helpers for buffers that other processes of the node map (CUDA IPC); not on the forward path.
int lloom_b200_peer_alloc(int64_t bytes, void **ptr) {
    if (!ptr || bytes <= 0) return LLOOM_ERR_NULL;
    cudaError_t e = cudaMalloc(ptr, (size_t)bytes);
    if (e == cudaSuccess) e = cudaMemset(*ptr, 0, (size_t)bytes);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return launch_status(e);
}
int lloom_b200_peer_free(void *ptr) { return launch_status(cudaFree(ptr)); }
int lloom_b200_peer_export(const void *ptr, unsigned char *handle64) {
    if (!ptr || !handle64) return LLOOM_ERR_NULL;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
    cudaIpcMemHandle_t h;
    cudaError_t e = cudaIpcGetMemHandle(&h, const_cast<void *>(ptr));
    if (e == cudaSuccess) memcpy(handle64, &h, 64);
    return launch_status(e);
}
int lloom_b200_peer_open(const unsigned char *handle64, void **ptr) {
    if (!ptr || !handle64) return LLOOM_ERR_NULL;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle64, 64);
    return launch_status(cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess));
}
int lloom_b200_peer_close(void *ptr) { return launch_status(cudaIpcCloseMemHandle(ptr)); }

int lloom_b200_qmatmul_fwd_static(int w_dtype, const void *w_blocks, const float *x, float *y, int64_t m, int64_t n,
                                  int64_t k, int64_t ldy, void *stream) {
    int rc = check_common(w_dtype, m, n, k);
    if (rc != LLOOM_OK) return rc;
    if (ldy < n) return LLOOM_ERR_SHAPE;
    if (!w_blocks || !x || !y) return LLOOM_ERR_NULL;
    if (!aligned(w_blocks, 16) || !aligned(x, 16) || !aligned(y, 4)) return LLOOM_ERR_ALIGN;
    if (m > 8 || m * lloom_b200_act_row_bytes(w_dtype, k) > (int64_t)LLOOM_B200_STATIC_SCRATCH_BYTES)
        return LLOOM_ERR_STATIC_LIMIT;
    void *scratch = nullptr;
    rc = static_scratch_ptr(&scratch);  // first call per device: cudaGetSymbolAddress (keep it out of captures)
    if (rc != LLOOM_OK) return rc;
    // The quantizer writes every byte of the m activation rows the GEMV then reads; the rest of the
    // array (left over from earlier calls) is never touched.
    rc = launch_status(launch_quantize_act(w_dtype, x, LLOOM_F32, m, k, scratch, default_io().overlap, (cudaStream_t)stream));
    if (rc != LLOOM_OK) return rc;
    return blocks_gemv(w_dtype, w_blocks, scratch, y, m, n, k, ldy, stream, default_io());
}

int lloom_b200_dequantize(int dtype, const void *blocks, int64_t elem_count, void *out, int out_is_f16,
                          void *stream) {
    if (!supported_weight(dtype)) return LLOOM_ERR_DTYPE;
    if (elem_count <= 0 || elem_count % lloom_b200_block_elems(dtype) != 0) return LLOOM_ERR_SHAPE;
    if (!blocks || !out) return LLOOM_ERR_NULL;
    if (!aligned(blocks, 16) || !aligned(out, 16)) return LLOOM_ERR_ALIGN;
    const unsigned grid = (unsigned)ceil_div64(elem_count / 8, 256);
    with_format(dtype, [&](auto fmt) {
        if (out_is_f16)
            dequantize_kernel<decltype(fmt)::value, true><<<grid, 256, 0, (cudaStream_t)stream>>>((const uint8_t *)blocks, elem_count, out);
        else
            dequantize_kernel<decltype(fmt)::value, false><<<grid, 256, 0, (cudaStream_t)stream>>>((const uint8_t *)blocks, elem_count, out);
    });
    return launch_status(cudaGetLastError());
}

int lloom_b200_get_rows(int dtype, const void *blocks, int64_t rows, int64_t hidden, const uint32_t *ids,
                        int64_t n_ids, float *out, void *stream) {
    return get_rows(dtype, blocks, rows, hidden, ids, false, n_ids, out, stream, default_io().overlap);
}

}  // extern "C"
