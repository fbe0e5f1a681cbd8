// Prefill GEMM for Q8_0, Q4_0, Q5_0 and Q6_K weights on tcgen05 tensor cores (sm_100a), exact-integer formulation.
//
//   Q8_0 x Q8_0 (k_quants.rs:800-818, avx.rs:71-87):     y[m,n] = sum over 32-element blocks b of (d_w[n,b]*d_a[m,b]) * dot32(q_w, q_a)
//   Q6_K x Q8_K (k_quants.rs:2115-2172, avx.rs:131-216):  y[m,n] = sum over superblocks b of (d_a[m,b]*d_w[n,b]) * S,
//                                                         S = sum_{j<16} sc_j * dot16(q6_j - 32, q8_j)
// through the m > 1 arm of k_quants::matmul (k_quants.rs:2518-2585).
//
// The block sums are integer contractions, so they run on the tensor cores (kind::f16, f32 accumulators in tensor
// memory) with every operand an integer that f16 represents exactly:
//   Q8_0: A = q_w, B = q_a (|.| <= 127); one accumulator drain per 32 of K, where the two f16 block scales meet.
//   Q4_0 / Q5_0 (k_quants.rs:320-392, 602-700; dotted with Q8_0 activations like Q8_0): the same with A = nibble - 8
//         / (nibble | fifth bit << 4) - 16; only the weight image and the place of the block scale differ.
//   Q6_K: v = sc_j * (q6 - 32) has up to 13 significant bits, so it is split v = hi + lo with lo = v mod 64 in
//         [0, 63] and hi a multiple of 64 in [-4096, 4032]: both exact in f16.  The two planes multiply the same
//         B = q8 codes and add into the same accumulator, which then holds S itself; one drain per 256 of K.
// The kernel is the Q4_K GEMM's frame (gemm_q4k.cuh) with the drain group, the plane count and the activation rows
// per tile (BM, the UMMA N) as parameters: 128 x BM output tile per CTA; operands arrive as ready-made
// 128-byte-swizzled K-major images by bulk copies; 512 / BM accumulators in tensor memory, so the drain of group g
// overlaps the MMAs of the following groups.  An MMA reads both operands from shared memory (8 KB per M = 128,
// N = 128, K = 16 instruction, 12 KB for twice the work at N = 256) and the bulk copies write as much again, so N = 256
// does more per byte: Q6_K (one drain per 256 of K) runs at BM = 256 unless smaller tiles fill the SMs better (gemm.cu); Q8_0 / Q4_0 / Q5_0 (one drain per 32 of K) are bound by their epilogue and stay at 128.
// Warp roles: 0-7 epilogue, 8 operand copies, 9 MMA issuer (one elected thread), 10 scale tiles (bulk copy of the
// activation scales; for the 32-of-K formats also the gather of the weight rows' f16 scales from the canonical blocks).
// The scale tiles travel in their own ring (a slot = 8 drain groups for the 32-of-K formats), released by the epilogue
// warps separately from the accumulators.  Epilogue of the 32-of-K formats: accumulators are read in the MMA fragment
// layout (tcgen05.ld.16x256b: 4 rows x 16 columns per thread), so a thread needs 16 + 4 scale words per group instead
// of 64 + 1; per output one exact product d_w * d_a and one fused multiply-add, the AVX2 arm's two operations.
// All waits are bounded and abortable; tensor memory is released on every path.
#pragma once

#include "gemm_q4k.cuh"

namespace lloom {

template <int GROUP_K, int PLANES, int BM>
struct PlanesCfg {
    static constexpr int kEpiWarps = 8;                // BM / 2 accumulator columns per warp (sixteen warps of BM / 4
                                                       // columns measured 1.6x slower on the 32-of-K formats)
    static constexpr int kGroupK = GROUP_K;            // K elements per accumulator drain
    static constexpr int kPlanes = PLANES;             // f16 images per weight element
    static constexpr int kBM = BM;                     // activation rows per tile (UMMA N): 128 or 256
    static constexpr int kStageK = PLANES == 1 ? 128 : 64;  // K elements per pipeline stage
    static constexpr int kStages = (PLANES == 1 || BM == 256) ? 3 : 4;
    static constexpr int kAtomsPerStage = kStageK / 64;
    static constexpr int kBAtomBytes = BM * 64 * 2;    // B atom: BM rows x 64 of K
    static constexpr int kStageABytes = kAtomsPerStage * PLANES * kGemmAtomBytes;
    static constexpr int kStageBBytes = kAtomsPerStage * kBAtomBytes;
    static constexpr int kAccBufs = 512 / BM;
    static constexpr int kDaBytes = BM * 4;             // activation scales of one drain group
    // The scale tiles travel in a ring of their own: a slot holds the scales of kDaGroups consecutive drain groups.
    // With a drain every 32 of K a slot covers eight groups, so a copy's trip to L2 is paid once per 256 of K and is
    // not on the path from one drain of an accumulator to its next use.
    static constexpr int kDaGroups = GROUP_K >= 256 ? 1 : 8;
    static constexpr int kDaSlots = GROUP_K >= 256 ? kAccBufs : 3;
    static constexpr int kDaSlotBytes = kDaGroups * kDaBytes;
    // Where a group is 32 of K the weight rows' scales ride in the same ring (gathered from the canonical blocks by the
    // scale warp, 128 f32 per group); where a group is 256 of K each epilogue thread fetches its row's scale itself.
    static constexpr bool kSmemW = GROUP_K < 256;
    static constexpr int kDwSlotBytes = kSmemW ? kDaGroups * kGemmBN * 4 : 0;
    // 64 or 128 running sums per epilogue thread beside the read-out; three whole warpgroups, so that the two epilogue
    // warpgroups can take registers from the third (setmaxnreg): epilogue, operand copies, MMA issuer, scale copies, idle
    static constexpr int kThreads = 384;
    // shared memory map (offsets from a 1024-byte aligned base)
    static constexpr int kOffA = 0;
    static constexpr int kOffB = kOffA + kStages * kStageABytes;
    static constexpr int kOffDa = kOffB + kStages * kStageBBytes;
    static constexpr int kOffDw = kOffDa + kDaSlots * kDaSlotBytes;
    static constexpr int kOffBars = kOffDw + kDaSlots * kDwSlotBytes;
    static constexpr int kNumBars = 2 * kStages + 2 * kAccBufs + 2 * kDaSlots;
    static constexpr int kOffMisc = kOffBars + kNumBars * 8;
    static constexpr int kSmemBytes = kOffMisc + 16 + 1024;  // + alignment slack
};

// Operand images: activation side [m-tile][k/64 atoms][BM x 128 B] + scales [m-tile][k/GROUP_K][BM] f32;
// weight side [n-tile][k/64 atoms][PLANES][16 KB].
struct PlanesActLayout {
    int64_t bimg, dat, total;
};
__host__ __device__ inline PlanesActLayout planes_act_layout(int64_t m, int64_t k, int group_k, int bm) {
    PlanesActLayout s;
    const int64_t mt = (m + bm - 1) / bm;
    s.bimg = 0;
    s.dat = mt * (k / 64) * bm * 128;
    s.total = (s.dat + mt * (k / group_k) * bm * 4 + 1023) / 1024 * 1024;
    return s;
}
__host__ __device__ inline int64_t planes_weight_bytes(int64_t n, int64_t k, int planes) {
    return (n + kGemmBN - 1) / kGemmBN * (k / 64) * planes * kGemmAtomBytes;
}

__device__ __forceinline__ uint32_t f16x2_from_ints(int a, int b) {
    const __half2 h = __halves2half2(__int2half_rn(a), __int2half_rn(b));
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Canonical activation blocks -> B image + scale plane.  One CTA per (m-tile, 64-element atom of K), one thread
// per activation row of the tile (BM threads).  ACT_Q8_0: 34-byte Q8_0 blocks (f16 d, 32 codes); else 292-byte Q8_K
// blocks (f32 d, 256 codes).
template <bool ACT_Q8_0, int BM>
__global__ void __launch_bounds__(BM) planes_prep_kernel(const uint8_t *__restrict__ act, int m, int k,
                                                         uint8_t *__restrict__ scratch) {
    launch_dependents();
    const int atoms = k / 64;
    const int mt = blockIdx.x / atoms, atom = blockIdx.x % atoms;
    const int t = threadIdx.x, row = mt * BM + t;
    const int group_k = ACT_Q8_0 ? 32 : 256;
    const PlanesActLayout lay = planes_act_layout(m, k, group_k, BM);
    uint8_t *img = scratch + lay.bimg + ((int64_t)mt * atoms + atom) * (BM * 128);
    float *dat = reinterpret_cast<float *>(scratch + lay.dat) + (int64_t)mt * (k / group_k) * BM;
    int q[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) q[i] = 0;
    if (row < m) {
        if (ACT_Q8_0) {
            const uint8_t *blk = act + ((int64_t)row * (k / 32) + atom * 2) * Q8_0_BYTES;  // 2-byte aligned
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned short *p16 = reinterpret_cast<const unsigned short *>(blk + h * Q8_0_BYTES);
                dat[(atom * 2 + h) * BM + t] = f16_bits_to_f32(p16[0]);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const unsigned short w = p16[1 + i];
                    q[h * 32 + 2 * i] = (int)(int8_t)(w & 0xff);
                    q[h * 32 + 2 * i + 1] = (int)(int8_t)(w >> 8);
                }
            }
        } else {
            const uint8_t *blk = act + ((int64_t)row * (k / 256) + (atom >> 2)) * Q8K_BYTES;  // 4-byte aligned
            if ((atom & 3) == 0) dat[(atom >> 2) * BM + t] = *reinterpret_cast<const float *>(blk);
            const uint32_t *p32 = reinterpret_cast<const uint32_t *>(blk + 4 + (atom & 3) * 64);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const uint32_t w = p32[i];
#pragma unroll
                for (int j = 0; j < 4; ++j) q[4 * i + j] = (int)(int8_t)(w >> (8 * j));
            }
        }
    } else {
        if (ACT_Q8_0) {
            dat[(atom * 2) * BM + t] = 0.0f;
            dat[(atom * 2 + 1) * BM + t] = 0.0f;
        } else if ((atom & 3) == 0) {
            dat[(atom >> 2) * BM + t] = 0.0f;
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint4 out = make_uint4(f16x2_from_ints(q[8 * c], q[8 * c + 1]), f16x2_from_ints(q[8 * c + 2], q[8 * c + 3]),
                                     f16x2_from_ints(q[8 * c + 4], q[8 * c + 5]), f16x2_from_ints(q[8 * c + 6], q[8 * c + 7]));
        *reinterpret_cast<uint4 *>(img + sw128_offset(t, 8 * c)) = out;
    }
}

// f32 activations -> the same B image + scale plane in one pass (the forward entries: no canonical blocks in between).
// One warp per (padded activation row, 256-element span of K), lane l holding elements 8l .. 8l + 7 of the span, i.e.
// one 16-byte chunk of the image; the quantizers are the warp functions of the stand-alone quantizer kernels, so the
// codes and scales are those of the canonical blocks bit for bit.  ACT_Q8_0: eight 32-element blocks per span (four
// lanes each; k may end in the middle of a span); else one Q8_K block.
template <bool ACT_Q8_0, int BM>
__global__ void __launch_bounds__(256) planes_prep_f32_kernel(const void *__restrict__ x, int x_type, int m, int k, uint8_t *__restrict__ scratch) {
    launch_dependents();
    const int spans = (k + 255) / 256, atoms = k / 64;
    const int lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);  // (padded row, span)
    const int64_t prow = item / spans;
    const int sp = (int)(item % spans);
    const int64_t mt = prow / BM;
    const int t = (int)(prow % BM);
    if (mt >= (m + BM - 1) / BM) return;  // whole warp
    const int group_k = ACT_Q8_0 ? 32 : 256;
    const PlanesActLayout lay = planes_act_layout(m, k, group_k, BM);
    const int e0 = sp * 256 + lane * 8;      // first of the lane's elements
    const bool in_k = e0 < k;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    if (prow < m && in_k) load8(x, x_type, prow * k + e0, v);  // rows of the last tile past m stay zero
    uint32_t q_lo = 0, q_hi = 0;
    float *dat = reinterpret_cast<float *>(scratch + lay.dat) + mt * (k / group_k) * BM;
    if (ACT_Q8_0) {
        unsigned short d16;
        q8_0_quantize_quad(v, q_lo, q_hi, d16);
        if (in_k && (lane & 3) == 0) dat[(int64_t)(sp * 8 + (lane >> 2)) * BM + t] = f16_bits_to_f32(d16);
    } else {
        float d;
        int sum16;
        q8k_quantize_warp(v, lane, q_lo, q_hi, d, sum16);
        if (lane == 0) dat[(int64_t)sp * BM + t] = d;
    }
    if (!in_k) return;
    auto cvt2 = [](uint32_t w, int sh) -> uint32_t {
        const __half2 h = __floats2half2_rn((float)(int)(int8_t)(w >> sh), (float)(int)(int8_t)(w >> (sh + 8)));
        return *reinterpret_cast<const uint32_t *>(&h);
    };
    const int atom = sp * 4 + (lane >> 3), e = (lane & 7) * 8;
    uint8_t *img = scratch + lay.bimg + (mt * atoms + atom) * (int64_t)(BM * 128);
    *reinterpret_cast<uint4 *>(img + sw128_offset(t, e)) = make_uint4(cvt2(q_lo, 0), cvt2(q_lo, 16), cvt2(q_hi, 0), cvt2(q_hi, 16));
}

// Weight blocks -> A image.  A thread writes one 16-byte chunk (eight elements) of a row of an atom per plane, eight lanes a
// whole 128-byte row, so that a warp stores whole lines (a thread per row, 16 bytes at a time into 32 rows at once: [4096, 14336] Q6_K with 512 rows
// took 282 us a call, this 228; [8192, 2048] Q8_0 with 1000 rows 183 and 154).  32 rows x two atoms per CTA; rows past the end are zero.
//   Q8_0: the codes; Q4_0 / Q5_0: nibble - 8, or (nibble | fifth bit << 4) - 16 (k_quants.rs:299-318, 578-600: low nibbles are
//   elements 0..15 of a block, high nibbles 16..31).
//   Q6_K: two planes, hi = v - (v mod 64) and lo = v mod 64 with v = sc_j * (q6 - 32) (k_quants.rs:2327-2358 for the codes).
template <int DTYPE>
__device__ __forceinline__ void expand_chunk(const uint8_t *row_blocks, int atom, int c, int (&v)[8]) {
    auto u16 = [](const uint8_t *p) { return (uint32_t)__ldg(reinterpret_cast<const unsigned short *>(p)); };
    auto load8b = [&](const uint8_t *p, uint32_t &a, uint32_t &b) {  // eight bytes, 2-byte aligned
        a = u16(p) | (u16(p + 2) << 16);
        b = u16(p + 4) | (u16(p + 6) << 16);
    };
    uint32_t w0, w1;
    if (DTYPE == LLOOM_Q8_0) {
        load8b(row_blocks + (int64_t)(atom * 2 + (c >> 2)) * Q8_0_BYTES + 2 + 8 * (c & 3), w0, w1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = (int)(int8_t)(w0 >> (8 * i));
            v[4 + i] = (int)(int8_t)(w1 >> (8 * i));
        }
    } else if (DTYPE == LLOOM_Q4_0 || DTYPE == LLOOM_Q5_0) {
        constexpr bool kFive = DTYPE == LLOOM_Q5_0;
        const uint8_t *blk = row_blocks + (int64_t)(atom * 2 + (c >> 2)) * (kFive ? Q5_0_BYTES : Q4_0_BYTES);
        const int cc = c & 3;  // elements 8cc .. 8cc + 7 of the block
        load8b(blk + (kFive ? 6 : 2) + 8 * (cc & 1), w0, w1);
        const int sh = cc & 2 ? 4 : 0;
        const uint32_t bits = kFive ? (u16(blk + 2) | (u16(blk + 4) << 16)) >> (8 * cc) : 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = (int)((i < 4 ? w0 : w1) >> (8 * (i & 3) + sh)) & 0xF;
            v[i] = kFive ? (q | (int)(((bits >> i) & 1u) << 4)) - 16 : q - 8;
        }
    } else {
        const uint8_t *blk = row_blocks + (int64_t)(atom >> 2) * Q6K_BYTES;
        const int a = atom & 3, h = a >> 1, gq = (a & 1) * 2 + (c >> 2), l = 8 * (c & 3);  // element 128h + 32gq + l ..
        uint32_t h0, h1;
        load8b(blk + 64 * h + (gq & 1) * 32 + l, w0, w1);
        load8b(blk + 128 + 32 * h + l, h0, h1);
        const int sc = (int)(int8_t)__ldg(blk + 192 + 8 * h + (l >> 4) + 2 * gq);
        const int sh = gq & 2 ? 4 : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t lo4 = ((i < 4 ? w0 : w1) >> (8 * (i & 3) + sh)) & 0xF, hi2 = ((i < 4 ? h0 : h1) >> (8 * (i & 3) + 2 * gq)) & 3;
            v[i] = sc * ((int)(lo4 | (hi2 << 4)) - 32);
        }
    }
}

template <int DTYPE>
__global__ void __launch_bounds__(256) planes_expand_kernel(const uint8_t *__restrict__ w, int64_t row_bytes, int n, int k,
                                                            uint8_t *__restrict__ image) {
    constexpr int kPlanes = DTYPE == LLOOM_Q6_K ? 2 : 1;
    launch_dependents();
    const int atoms = k / 64, pairs = atoms / 2;
    const int tile_pair = blockIdx.x >> 2, nt = tile_pair / pairs, atom0 = (tile_pair - nt * pairs) * 2;
    const int r = (blockIdx.x & 3) * 32 + (threadIdx.x >> 3), c = threadIdx.x & 7;
    const int64_t row = (int64_t)nt * kGemmBN + r;
    int v[2][8];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        if (row < n) expand_chunk<DTYPE>(w + row * row_bytes, atom0 + a, c, v[a]);
        else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[a][i] = 0;
        }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        uint8_t *img = image + ((int64_t)nt * atoms + atom0 + a) * kPlanes * kGemmAtomBytes + sw128_offset(r, 8 * c);
        auto store = [](uint8_t *dst, const int (&x)[8]) {
            *reinterpret_cast<uint4 *>(dst) = make_uint4(f16x2_from_ints(x[0], x[1]), f16x2_from_ints(x[2], x[3]), f16x2_from_ints(x[4], x[5]),
                                                         f16x2_from_ints(x[6], x[7]));
        };
        if (kPlanes == 1) {
            store(img, v[a]);
        } else {
            int lo[8], hi[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                lo[i] = v[a][i] & 63;
                hi[i] = v[a][i] - lo[i];
            }
            store(img, hi);
            store(img + kGemmAtomBytes, lo);
        }
    }
    wait_predecessor();  // the GEMM waits for this kernel only, which therefore ends after the activation side has
}

// 16 lanes x 64 columns of tensor memory as the MMA accumulator fragment: thread T = 4*g + c holds, for each block i of
// eight columns, v[4i], v[4i+1] = lane g, columns 8i + 2c, 8i + 2c + 1 and v[4i+2], v[4i+3] = lane g + 8, same columns.
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

struct PlanesParams {
    const uint8_t *w;        // canonical weight blocks of the launch's rows (for the per-group f16 scales)
    const uint8_t *act_img;  // planes_prep_kernel output
    const uint8_t *w_img;    // expand kernel output
    void *y;                 // outputs of type y_type
    int y_type;
    int64_t ldy;
    int64_t row_bytes;
    int m, n_end, k;  // n_end: rows of the launch (rows >= n_end are masked)
    int n_tiles, m_tiles;
    int scale_stride, scale_off;  // weight scale of group g of a row: f16 at row + g * scale_stride + scale_off
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::kThreads, 1) gemm_planes_kernel(const PlanesParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Cfg::kOffBars);
    uint64_t *full = bars, *empty = bars + Cfg::kStages;
    uint64_t *acc_full = bars + 2 * Cfg::kStages, *acc_empty = acc_full + Cfg::kAccBufs;
    uint64_t *da_full = acc_empty + Cfg::kAccBufs, *da_empty = da_full + Cfg::kDaSlots;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + Cfg::kOffMisc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::kOffMisc + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // m-tiles of one n-tile are neighbours in launch order, so the n-tile's A images are shared through L2
    const int mt = blockIdx.x % p.m_tiles, nt = blockIdx.x / p.m_tiles;
    const int m0 = mt * Cfg::kBM;
    const int64_t n0 = (int64_t)nt * kGemmBN;
    const int atoms = p.k / 64;
    const int ngroups = p.k / Cfg::kGroupK;
    const int nstages = p.k / Cfg::kStageK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < Cfg::kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < Cfg::kAccBufs; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], Cfg::kEpiWarps);
        }
        for (int i = 0; i < Cfg::kDaSlots; ++i) {
            mbar_init(&da_full[i], Cfg::kSmemW ? 2 : 1);  // the copy's bytes (+ the gathered weight scales)
            mbar_init(&da_empty[i], Cfg::kEpiWarps);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == Cfg::kEpiWarps + 1) {  // tensor memory: all 512 columns, 512 / BM accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    wait_predecessor();  // the operand images are there

    // Per scheduler: two epilogue warps of 216 registers and one other warp of 72.  One setmaxnreg per
    // warpgroup, executed by all of its warps at the top of the branch that holds all of the warpgroup's code.
    if (warp < Cfg::kEpiWarps) {
        // ------------------------------ epilogue ------------------------------
        // warp w: TMEM lanes 32*(w%4).. (hardware rule), accumulator columns (BM/2)*(w/4)..
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;" ::: "memory");
        constexpr int kCW = Cfg::kBM / (Cfg::kEpiWarps / 4);  // columns per warp
        const int q = warp & 3, half = warp >> 2;
        if (Cfg::kSmemW) {
            // A drain every 32 of K: the scales, not the sums, set the cost.  With a tensor-memory lane per thread every
            // thread would fetch all 64 activation scales of its columns for every group (the same words in all 32
            // lanes, 64 shared-memory wavefronts per warp and group); in the accumulator-fragment layout a thread
            // holds 4 rows x 16 columns, so it needs 16 activation scales and 4 weight scales (20 wavefronts).
            const int fg = lane >> 2, fc = lane & 3;
            float acc[4][16];  // [row j: 32q + fg + 8j][2i + e: column 64*half + 8i + 2fc + e]
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[j][i] = 0.0f;
            // Rows 0-15 of the warp's lane quarter (va) and rows 16-31 (vb) take turns: while one half's sums are scaled and
            // added, the other half -- behind vb the first half of the next group -- is on its way from tensor memory
            // ([8192, 2048] Q8_0, 1000 rows, prebuilt image: 138 us, 144 with both halves waited for first).
            // k is a multiple of 128, so groups come in fours, one per accumulator.
            static_assert(!Cfg::kSmemW || (Cfg::kAccBufs == 4 && Cfg::kDaGroups % 4 == 0), "four groups per turn of the accumulators");
            const uint32_t t_main = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * kCW);
            uint32_t va[32], vb[32];
            bool ok = mbar_wait_abortable<64>(&acc_full[0], 0, abort_flag);
            tc_fence_after();
            if (ok) tmem_ld_frag64(t_main, va);
            int slot = 0;
            uint32_t slot_par = 0, par = 0;
            for (int g0 = 0; g0 < ngroups && ok; g0 += Cfg::kDaGroups) {
                ok = mbar_wait_abortable<64>(&da_full[slot], slot_par, abort_flag);
                const float *dws = reinterpret_cast<const float *>(smem + Cfg::kOffDw + slot * Cfg::kDwSlotBytes) + q * 32 + fg;
                const float2 *das = reinterpret_cast<const float2 *>(smem + Cfg::kOffDa + slot * Cfg::kDaSlotBytes + half * kCW * 4) + fc;
                const int g1 = min(g0 + Cfg::kDaGroups, ngroups);
                for (int g = g0; g < g1 && ok; g += 4, par ^= 1) {
#pragma unroll
                    for (int buf = 0; buf < 4; ++buf, dws += kGemmBN, das += Cfg::kDaBytes / 8) {
                        if (!ok) break;
                        float dw[4];
                        float2 da2[8];
#pragma unroll
                        for (int j = 0; j < 4; ++j) dw[j] = dws[8 * j];
#pragma unroll
                        for (int i = 0; i < 8; ++i) da2[i] = das[4 * i];
                        // scalar multiplies and fused multiply-adds: they issue on both FMA pipes, the packed f32x2 forms on one
                        auto add = [&](int j0, const uint32_t (&v)[32]) {
#pragma unroll
                            for (int j = j0; j < j0 + 2; ++j)
#pragma unroll
                                for (int i = 0; i < 8; ++i) {
                                    const int ix = 4 * i + 2 * (j & 1);
                                    acc[j][2 * i] = __fmaf_rn(__fmul_rn(da2[i].x, dw[j]), __uint_as_float(v[ix]), acc[j][2 * i]);
                                    acc[j][2 * i + 1] = __fmaf_rn(__fmul_rn(da2[i].y, dw[j]), __uint_as_float(v[ix + 1]), acc[j][2 * i + 1]);
                                }
                        };
                        tmem_ld_wait();
                        loaded(va);
                        tmem_ld_frag64(t_main + (uint32_t)(buf * Cfg::kBM) + (16u << 16), vb);
                        add(0, va);
                        tmem_ld_wait();
                        loaded(vb);
                        // everything this warp needs from this accumulator is in registers now
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&acc_empty[buf]);
                        if (buf < 3 || g + 4 < ngroups) {
                            ok = mbar_wait_abortable<64>(&acc_full[(buf + 1) & 3], buf < 3 ? par : par ^ 1, abort_flag);
                            if (!ok) break;
                            tc_fence_after();
                            tmem_ld_frag64(t_main + (uint32_t)(((buf + 1) & 3) * Cfg::kBM), va);
                        }
                        add(2, vb);
                    }
                }
                // the slot is rewritten by a bulk copy (async proxy) right after the arrivals, so this warp's reads of it
                // (generic proxy) are fenced first
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&da_empty[slot]);
                if (++slot == Cfg::kDaSlots) {
                    slot = 0;
                    slot_par ^= 1;
                }
            }
            if (ok) with_y_type(p.y, p.y_type, [&](auto *y) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int64_t n = n0 + q * 32 + fg + 8 * j;
                    if (n >= p.n_end) continue;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int mrow = m0 + half * kCW + 8 * i + 2 * fc;
                        if (mrow < p.m) put_y(y, (int64_t)mrow * p.ldy + n, acc[j][2 * i]);
                        if (mrow + 1 < p.m) put_y(y, (int64_t)(mrow + 1) * p.ldy + n, acc[j][2 * i + 1]);
                    }
                }
            });
        } else {
        const int r = q * 32 + lane;  // row of the tile == TMEM lane
        const int64_t n = n0 + r;
        const bool row_ok = n < p.n_end;
        const uint8_t *wrow = p.w + (row_ok ? n : 0) * p.row_bytes + p.scale_off;
        uint64_t out2[kCW / 2];
#pragma unroll
        for (int j = 0; j < kCW / 2; ++j) out2[j] = 0ull;
        // group >= 256 of K: the row's weight scale of the next group is fetched while this group is drained
        unsigned short hdr_nxt = 0;
        if (row_ok) hdr_nxt = __ldg(reinterpret_cast<const unsigned short *>(wrow));
        bool ok = true;
        for (int g = 0; g < ngroups && ok; ++g) {
            const int buf = g % Cfg::kAccBufs;
            const uint32_t par = (g / Cfg::kAccBufs) & 1;
            const int slot_i = g / Cfg::kDaGroups, in_slot = g % Cfg::kDaGroups, slot = slot_i % Cfg::kDaSlots;
            if (in_slot == 0) ok = mbar_wait_abortable<64>(&da_full[slot], (slot_i / Cfg::kDaSlots) & 1, abort_flag);
            if (!ok) break;
            const float dw = f16_bits_to_f32(hdr_nxt);
            if (row_ok && g + 1 < ngroups)
                hdr_nxt = __ldg(reinterpret_cast<const unsigned short *>(wrow + (int64_t)(g + 1) * p.scale_stride));
            const uint64_t dw2 = pack2f(dw, dw);
            ok = mbar_wait_abortable<64>(&acc_full[buf], par, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t t_main = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * Cfg::kBM + half * kCW);
            // the activation scales of this warp's columns, as f32 pairs, times the weight scale: (d_a * d_w)
            const ulonglong2 *dap = reinterpret_cast<const ulonglong2 *>(smem + Cfg::kOffDa + slot * Cfg::kDaSlotBytes +
                                                                         in_slot * Cfg::kDaBytes + half * kCW * 4);
#pragma unroll
            for (int c = 0; c < kCW / 64; ++c) {  // 64 columns at a time: two loads in flight
                uint32_t va[32], vb[32];
                tmem_ld32(t_main + 64 * c, va);
                tmem_ld32(t_main + 64 * c + 32, vb);
                uint64_t d2[16];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const ulonglong2 t = dap[16 * c + j];
                    d2[2 * j] = mul_f32x2(t.x, dw2);
                    d2[2 * j + 1] = mul_f32x2(t.y, dw2);
                }
                tmem_ld_wait();
                loaded(va);
                loaded(vb);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    out2[32 * c + j] = fma_f32x2(d2[j], (uint64_t)va[2 * j] | ((uint64_t)va[2 * j + 1] << 32), out2[32 * c + j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const ulonglong2 t = dap[16 * c + 8 + j];
                    d2[2 * j] = mul_f32x2(t.x, dw2);
                    d2[2 * j + 1] = mul_f32x2(t.y, dw2);
                }
                if (c == kCW / 64 - 1) {
                    // everything this warp needs from tensor memory and from the scale tiles is in registers now
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[buf]);
                    if (in_slot == Cfg::kDaGroups - 1 || g == ngroups - 1) {
                        // the slot is rewritten by a bulk copy (async proxy) right after the arrivals, so this warp's
                        // reads of it (generic proxy) are fenced first
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&da_empty[slot]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    out2[32 * c + 16 + j] = fma_f32x2(d2[j], (uint64_t)vb[2 * j] | ((uint64_t)vb[2 * j + 1] << 32), out2[32 * c + 16 + j]);
            }
        }
        if (ok && row_ok) with_y_type(p.y, p.y_type, [&](auto *y) {
#pragma unroll
            for (int j = 0; j < kCW / 2; ++j) {
                const int mrow = m0 + half * kCW + 2 * j;
                if (mrow < p.m) put_y(y, (int64_t)mrow * p.ldy + n, __uint_as_float((uint32_t)(out2[j] & 0xffffffffu)));
                if (mrow + 1 < p.m) put_y(y, (int64_t)(mrow + 1) * p.ldy + n, __uint_as_float((uint32_t)(out2[j] >> 32)));
            }
        });
        }
    } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;" ::: "memory");
    if (warp == Cfg::kEpiWarps) {
        // ------------------------------ operand tiles: bulk copies ------------------------------
        // The whole warp walks the loop (lanes stay converged); lane 0 issues the copies.
        const uint8_t *aimg = p.w_img + (int64_t)nt * atoms * Cfg::kPlanes * kGemmAtomBytes;
        const uint8_t *bimg = p.act_img + (int64_t)mt * atoms * Cfg::kBAtomBytes;
        bool ok = true;
        for (int it = 0; it < nstages && ok; ++it) {
            const int s = it % Cfg::kStages;
            if (it >= Cfg::kStages) ok = mbar_wait_abortable<32>(&empty[s], ((it / Cfg::kStages) - 1) & 1, abort_flag);
            if (!ok) break;
            if (lane == 0) {
                mbar_arrive_expect_tx(&full[s], Cfg::kStageABytes + Cfg::kStageBBytes);
                bulk_g2s(smem + Cfg::kOffA + s * Cfg::kStageABytes, aimg + (int64_t)it * Cfg::kStageABytes, Cfg::kStageABytes, &full[s]);
                bulk_g2s(smem + Cfg::kOffB + s * Cfg::kStageBBytes, bimg + (int64_t)it * Cfg::kStageBBytes, Cfg::kStageBBytes, &full[s]);
            }
            __syncwarp();
        }
    } else if (warp == Cfg::kEpiWarps + 2) {
        // ------------------------------ activation scales, a slot of drain groups at a time ------------------------------
        const PlanesActLayout lay = planes_act_layout(p.m, p.k, Cfg::kGroupK, Cfg::kBM);
        const uint8_t *dat = p.act_img + lay.dat + (int64_t)mt * ngroups * Cfg::kDaBytes;
        const int nslots = (ngroups + Cfg::kDaGroups - 1) / Cfg::kDaGroups;
        bool ok = true;
        for (int si = 0; si < nslots && ok; ++si) {
            const int slot = si % Cfg::kDaSlots;
            if (si >= Cfg::kDaSlots) ok = mbar_wait_abortable<32>(&da_empty[slot], ((si / Cfg::kDaSlots) - 1) & 1, abort_flag);
            if (!ok) break;
            if (lane == 0) {
                const int groups = min(Cfg::kDaGroups, ngroups - si * Cfg::kDaGroups);
                const uint32_t bytes = (uint32_t)(groups * Cfg::kDaBytes);
                mbar_arrive_expect_tx(&da_full[slot], bytes);
                bulk_g2s(smem + Cfg::kOffDa + slot * Cfg::kDaSlotBytes, dat + (int64_t)si * Cfg::kDaSlotBytes, bytes, &da_full[slot]);
            }
            if (Cfg::kSmemW) {
                // the f16 scales of the tile's 128 weight rows for the slot's groups: lane l gathers rows l, l + 32, ...
                const int groups = min(Cfg::kDaGroups, ngroups - si * Cfg::kDaGroups);
                float *dws = reinterpret_cast<float *>(smem + Cfg::kOffDw + slot * Cfg::kDwSlotBytes);
#pragma unroll
                for (int j = 0; j < kGemmBN / 32; ++j) {
                    const int rr = lane + 32 * j;
                    const bool rok = n0 + rr < p.n_end;
                    const uint8_t *wp = p.w + (rok ? n0 + rr : 0) * p.row_bytes + p.scale_off +
                                        (int64_t)si * Cfg::kDaGroups * p.scale_stride;
                    unsigned short h[Cfg::kDaGroups];
#pragma unroll
                    for (int gi = 0; gi < Cfg::kDaGroups; ++gi)
                        h[gi] = (rok && gi < groups) ? __ldg(reinterpret_cast<const unsigned short *>(wp + (int64_t)gi * p.scale_stride))
                                                     : (unsigned short)0;
#pragma unroll
                    for (int gi = 0; gi < Cfg::kDaGroups; ++gi) dws[gi * kGemmBN + rr] = f16_bits_to_f32(h[gi]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&da_full[slot]);
            }
            __syncwarp();
        }
    } else if (warp == Cfg::kEpiWarps + 1) {
        // ------------------------------ MMA issuer: one elected thread (gemm_q4k.cuh) ------------------------------
        if (elect_one()) {
            // instruction descriptor: D = f32, A = B = f16, both K-major, N = BM, M = 128
            const uint32_t idesc = (1u << 4) | ((uint32_t)(Cfg::kBM >> 3) << 17) | ((uint32_t)(kGemmBN >> 4) << 24);
            const uint32_t a_lo0 = umma_desc_lo(smem_u32(smem + Cfg::kOffA), 16), b_lo0 = umma_desc_lo(smem_u32(smem + Cfg::kOffB), 16);
            constexpr int kStepsPerStage = Cfg::kStageK / 16;
            constexpr int kStepsPerGroup = Cfg::kGroupK / 16;
            // a stage is one turn of the accumulators (32-of-K formats), or a part of one accumulator's group
            constexpr bool kTurn = Cfg::kStageK == Cfg::kGroupK * Cfg::kAccBufs;
            constexpr int kStagesPerGroup = kTurn ? 1 : Cfg::kGroupK / Cfg::kStageK;
            static_assert(kTurn || Cfg::kGroupK % Cfg::kStageK == 0, "stages and drain groups");
            bool ok = true;
            int s = 0, in_group = 0, acc = 0;      // stage slot; !kTurn: stage of the group, accumulator
            uint32_t full_par = 0, acc_par = 1;    // the accumulators' first use finds them empty
            for (int it = 0; it < nstages && ok; ++it) {
                ok = mbar_wait_abortable<0>(&full[s], full_par, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_lo = a_lo0 + (uint32_t)(s * (Cfg::kStageABytes >> 4));
                const uint32_t b_lo = b_lo0 + (uint32_t)(s * (Cfg::kStageBBytes >> 4));
#pragma unroll
                for (int kk = 0; kk < kStepsPerStage; ++kk) {  // K = 16 per instruction: atom kk/4, 32 bytes along its swizzled row
                    const int buf = kTurn ? kk / kStepsPerGroup : acc;
                    const bool first = kTurn ? kk % kStepsPerGroup == 0 : kk == 0 && in_group == 0;
                    if (first) {
                        ok = mbar_wait_abortable<0>(&acc_empty[buf], acc_par, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const uint32_t d_acc = tmem_base + (uint32_t)(buf * Cfg::kBM);
                    const uint32_t boff = (uint32_t)((kk >> 2) * (Cfg::kBAtomBytes >> 4) + (kk & 3) * 2);
#pragma unroll
                    for (int pl = 0; pl < Cfg::kPlanes; ++pl) {
                        const uint32_t aoff = (uint32_t)(((kk >> 2) * Cfg::kPlanes + pl) * (kGemmAtomBytes >> 4) + (kk & 3) * 2);
                        if (pl != 0 || kk % (kTurn ? kStepsPerGroup : kStepsPerStage) != 0) umma_f16_lo<true>(d_acc, a_lo + aoff, b_lo + boff, idesc);
                        else if (kTurn) umma_f16_lo<false>(d_acc, a_lo + aoff, b_lo + boff, idesc);
                        else umma_f16_lo_rt(d_acc, a_lo + aoff, b_lo + boff, idesc, in_group != 0 ? 1u : 0u);
                    }
                    if (kTurn && kk % kStepsPerGroup == kStepsPerGroup - 1) umma_commit(&acc_full[buf]);
                }
                if (!ok) break;
                umma_commit(&empty[s]);
                if (kTurn) {
                    acc_par ^= 1;
                } else if (++in_group == kStagesPerGroup) {
                    umma_commit(&acc_full[acc]);
                    in_group = 0;
                    if (++acc == Cfg::kAccBufs) {
                        acc = 0;
                        acc_par ^= 1;
                    }
                }
                if (++s == Cfg::kStages) {
                    s = 0;
                    full_par ^= 1;
                }
            }
        }
        __syncwarp();
    }
    }
    // ------------------------------ teardown ------------------------------
    tc_fence_before();
    __syncthreads();
    if (warp == Cfg::kEpiWarps + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

}  // namespace lloom
