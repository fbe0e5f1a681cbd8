// Skinny product (2 to 128 activation rows, more where no tcgen05 GEMM exists) over canonical GGUF block rows, on the integer tensor cores.
//
// One warp-level `mma.sync.m16n8k32.s8` multiplies a 16-row x 32-element weight sub-block, unpacked to int8 in registers,
// by the 32 x 8 block of activation codes: exact int32 sums for 16 weight rows x 8 activation rows.  Weights are read
// packed, so a call streams 0.56 to 1.06 bytes per weight and writes nothing but its result; the tcgen05 GEMMs, which
// need the weights expanded to f16 operand images (1.9 to 4.9 times the packed bytes, written and read back), take over
// where their higher rate pays for that.
//
//   Q4_K / Q5_K (k_quants.rs:1540-1620, 1795-1880): the 6-bit sub-block scale multiplies the four accumulators as an
//     integer, so the superblock sum stays exact; the min term sum_j m_j * bsum_j is one f16 MMA over the sixteen
//     16-element sums (m_j <= 63, |bsum| <= 2032: exact); two f32 scales once per superblock, as in the reference.
//   Q6_K (k_quants.rs:2115-2172): scales per 16 elements, so m16n8k16 MMAs, else like Q4_K without the min term.
//   Q8_0 / Q4_0 / Q5_0 (k_quants.rs:800-818, 371-391, 500-513): a sum per 32-element block.  The accumulator starts at the
//     bit pattern of 1.5 * 2^23 (less the code offset times the block's sum of activation codes), so that the finished sum
//     read as a float is 1.5 * 2^23 + dot: one subtraction instead of an int -> float conversion, exact for |dot| < 2^22.
//
// What an MMA costs here: 8.5 cycles of its scheduler per m16n8k32 or m16n8k16 (measured, 16 warps), during which the
// scheduler issues nothing else.  A 16-row x 256-element tile is about 290 (Q4_K) to 580 (Q6_K) scheduler cycles for
// eight activation rows, 175 to 280 for every further eight.
//
// Frame: a CTA owns a contiguous range of 16-row tiles (and, past 48 activation rows, one of several groups of them,
// blockIdx.y).  It works on TR tiles at a time with TR x S x TN consumer warps: warp (tile, slot, column part) takes
// superblocks slot, slot + S, ... of its tile and part of the 8-row activation tiles.  A producer warp streams stages of
// S superblocks (eight where a warp keeps two sums) of TR x 16 rows by tiled TMA loads (rows `row_pitch` bytes apart:
// fragment loads hit distinct banks), and, unless they stay resident in shared memory, the same superblocks of the activations as
// one bulk copy.  The partial sums of an output meet in shared memory.  How many there are depends on k and the batch alone
// and the order of the additions is the dp4a kernel's (add_round), so a row's bits do not depend on the shard, the launch or (up
// to sixteen rows) the batch.
//
// Activations come as an image in fragment order (launch_quantize_image), per group of activation tiles
// [superblock][tile of T rows] units; T = 8, or 1 for a single row (the MMAs' other columns then repeat it and are
// dropped).  A unit:
//   codes  [4][row][tig][16 B]: what lane (gid = row, tig) feeds to the MMAs of a 64-element stretch
//   k-quants: sums [row][tig][8 B], the 16-element sums as f16 in the order of the f16 MMA's B fragment; d [row] f32
//   32-element formats: d [block][row] f32; Q4_0 / Q5_0: accumulator starts [block][row] int32
// Every fragment load is one conflict-free 16- or 8-byte load.
#pragma once

#include <cuda.h>

#include "gemv.cuh"

namespace lloom {

__device__ __forceinline__ void mma_s8_k32(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// unsigned weight bytes
__device__ __forceinline__ void mma_u8_k32(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same with another accumulator start: c = a * b + init
__device__ __forceinline__ void mma_s8_k32_from(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int init0, int init1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %10, %11};\n"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(init0), "r"(init1));
}
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};\n"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b));
}
__device__ __forceinline__ void mma_f16_k16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- activation image ----

// Where 4-byte word c (elements 4c .. 4c + 3) of a superblock of activation row t (of T) goes inside its unit: the lane
// (t, tig) that feeds it, and the word of that lane's 16 bytes.
__host__ __device__ inline int image_code_offset(int kind, int T, int t, int c) {
    if (kind == kImgQ6K) {  // element 128h + 32gq + 16s + 4tig + i: stretch 2h + s, word gq
        const int h = c >> 5, gq = (c >> 3) & 3, s = (c >> 2) & 1, tig = c & 3;
        return (2 * h + s) * 64 * T + (t * 4 + tig) * 16 + gq * 4;
    }
    const int g = c >> 4, half = (c >> 3) & 1, w = c & 7;  // 64-element stretch, its 32-element half, word of the half
    // Q4_0 / Q5_0 codes: words w and w + 4 come out of the same nibble bytes; else words 2tig and 2tig + 1 are neighbours
    const int tig = kind == kImgSplit ? (w & 3) : (w >> 1), pos = kind == kImgSplit ? (w >> 2) : (w & 1);
    return g * 64 * T + (t * 4 + tig) * 16 + half * 8 + pos * 4;
}
// offsets in a unit, times T; k-quants, and the 32-element formats
constexpr int kImgSums = 256, kImgKD = 288;
constexpr int kImgD = 256, kImgStart = 288;
constexpr int kMagicBits = 0x4B400000;                  // 1.5 * 2^23
constexpr float kMagic = 12582912.0f;

// One warp writes superblock `sb` of activation row t of a unit from the row's values (lane l: elements 8l .. 8l + 7).
__device__ __forceinline__ void values_to_image(const float (&v)[8], uint8_t *unit, int kind, int offset, int T, int t, int lane, bool in_k) {
    uint32_t q_lo, q_hi;
    if (kind == kImgK || kind == kImgQ6K) {
        float d;
        int sum16;
        q8k_quantize_warp(v, lane, q_lo, q_hi, d, sum16);
        const int next = __shfl_down_sync(0xffffffffu, sum16, 2);
        if ((lane & 3) == 0) {  // sums 2q and 2q + 1 (q = lane / 4): words q of the B fragment, second half from q = 4
            const int q = lane >> 2;
            const __half2 h = __floats2half2_rn((float)sum16, (float)next);
            *reinterpret_cast<__half2 *>(unit + kImgSums * T + (t * 4 + (q & 3)) * 8 + (q >> 2) * 4) = h;
        }
        if (lane == 0) *reinterpret_cast<float *>(unit + kImgKD * T + t * 4) = d;
    } else {
        unsigned short d16;
        q8_0_quantize_quad(v, q_lo, q_hi, d16);
        int s = __dp4a((int)q_lo, 0x01010101, __dp4a((int)q_hi, 0x01010101, 0));
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (in_k && (lane & 3) == 0) {
            const int blk = lane >> 2;
            *reinterpret_cast<float *>(unit + kImgD * T + (blk * T + t) * 4) = f16_bits_to_f32(d16);
            if (kind == kImgSplit) *reinterpret_cast<int *>(unit + kImgStart * T + (blk * T + t) * 4) = kMagicBits - offset * s;
        }
    }
    if (in_k) {
        *reinterpret_cast<uint32_t *>(unit + image_code_offset(kind, T, t, 2 * lane)) = q_lo;
        *reinterpret_cast<uint32_t *>(unit + image_code_offset(kind, T, t, 2 * lane + 1)) = q_hi;
    }
}

// f32 / f16 / bf16 activations -> the image; one warp per (padded activation row, superblock).  Rows past m are zero.
// In a chain of forwards its CTAs become resident beside the product in front (and wait there) if an SM has room for one:
// the seventeen warps of a product leave one of the four schedulers 1024 registers, a warp of 32 registers a thread, so CTAs
// of four such warps fit and eight do not (graph of Q4_K launches, 8 rows: [4096, 4096] 8.8 -> 5.4 us a forward, [4096, 14336]
// 13.8 -> 10.4, [14336, 4096] 14.0 -> 12.3; a layer's seven matmuls 67.6 -> 55.0).
constexpr int kQuantThreads = 128;
static __global__ void __launch_bounds__(kQuantThreads, 16) quantize_image_kernel(const void *__restrict__ x, int x_type, uint8_t *__restrict__ img,
                                                                    int kind, int offset, int unit_bytes, int m, int k, int ntiles,
                                                                    int group_nt, int T) {  // ntiles: whole groups
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the product may start streaming weights
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int nsb = (k + 255) >> 8, lane = threadIdx.x & 31;
    const int item = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);  // (row, superblock)
    const int row = item / nsb, sb = item - row * nsb;
    const int tile = row / T;
    if (tile >= ntiles) return;  // whole warp
    const int tg = tile / group_nt;
    uint8_t *unit = img + (((int64_t)tg * nsb + sb) * group_nt + (tile - tg * group_nt)) * unit_bytes;
    const int e0 = sb * 256 + lane * 8;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    if (row < m && e0 < k) load8(x, x_type, (int64_t)row * k + e0, v);
    values_to_image(v, unit, kind, offset, T, row - tile * T, lane, e0 < k);
}

// Canonical activation blocks -> the image (entries that are given blocks): in shared memory for up to eight rows
// (group_nt = 1), or in global memory.  Rows past m are left as they are: their columns are computed on whatever is there
// and never stored.
__device__ __forceinline__ void blocks_to_image(const uint8_t *act, uint8_t *img, int kind, int offset, int unit_bytes, int m, int k,
                                                int group_nt, int T, int64_t tid, int64_t nthreads) {
    const int nsb = (k + 255) >> 8;
    auto unit_of = [&](int row, int sb) {
        const int tile = row / T, tg = tile / group_nt;
        return img + (((int64_t)tg * nsb + sb) * group_nt + (tile - tg * group_nt)) * unit_bytes;
    };
    if (kind == kImgK || kind == kImgQ6K) {
        const int words = Q8K_BYTES / 4;
        const int64_t total = (int64_t)m * nsb * words;
        const uint32_t *src = reinterpret_cast<const uint32_t *>(act);
        for (int64_t i = tid; i < total; i += nthreads) {
            const uint32_t v = __ldg(src + i);
            const int blk = (int)(i / words), w = (int)(i - (int64_t)blk * words);
            const int row = blk / nsb, t = row % T;
            uint8_t *unit = unit_of(row, blk - row * nsb);
            if (w == 0) {
                *reinterpret_cast<uint32_t *>(unit + kImgKD * T + t * 4) = v;
            } else if (w <= 64) {
                *reinterpret_cast<uint32_t *>(unit + image_code_offset(kind, T, t, w - 1)) = v;
            } else {
                const int q = w - 65;  // 16-element sums 2q, 2q + 1
                const __half2 h = __floats2half2_rn((float)(short)(v & 0xffffu), (float)(short)(v >> 16));
                *reinterpret_cast<__half2 *>(unit + kImgSums * T + (t * 4 + (q & 3)) * 8 + (q >> 2) * 4) = h;
            }
        }
    } else {
        const int nblk = k >> 5;
        const int64_t total = (int64_t)m * nblk * 8;  // a thread per code word
        for (int64_t i = tid; i < total; i += nthreads) {
            const int blk = (int)(i >> 3), w = (int)(i & 7);
            const int row = blk / nblk, b = blk - row * nblk, t = row % T;
            const unsigned short *p = reinterpret_cast<const unsigned short *>(act + (int64_t)blk * Q8_0_BYTES);
            uint8_t *unit = unit_of(row, b >> 3);
            const uint32_t v = (uint32_t)__ldg(p + 1 + 2 * w) | ((uint32_t)__ldg(p + 2 + 2 * w) << 16);
            *reinterpret_cast<uint32_t *>(unit + image_code_offset(kind, T, t, (b & 7) * 8 + w)) = v;
            if (w == 0) {
                *reinterpret_cast<float *>(unit + kImgD * T + ((b & 7) * T + t) * 4) = f16_bits_to_f32(__ldg(p));
                if (kind == kImgSplit) {
                    int s = 0;
                    for (int j = 1; j <= 16; ++j) {
                        const unsigned short c = __ldg(p + j);
                        s += (int)(int8_t)(c & 0xff) + (int)(int8_t)(c >> 8);
                    }
                    *reinterpret_cast<int *>(unit + kImgStart * T + ((b & 7) * T + t) * 4) = kMagicBits - offset * s;
                }
            }
        }
    }
}

static __global__ void __launch_bounds__(256) blocks_to_image_kernel(const uint8_t *__restrict__ act, uint8_t *__restrict__ img, int kind,
                                                                     int offset, int unit_bytes, int m, int k, int group_nt, int T) {
    blocks_to_image(act, img, kind, offset, unit_bytes, m, k, group_nt, T, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
                    (int64_t)gridDim.x * blockDim.x);
}

// ---- formats: one superblock (nblk 32-element blocks of it, for the 32-element formats) of a 16-row tile ----
// ra / rb: the superblock of rows gid and gid + 8 in shared memory; act: the activation unit of the first tile, the next
// `u.bytes` on.  out[nt] = (row gid, column 2tig), (gid, 2tig + 1), (gid + 8, 2tig), (gid + 8, 2tig + 1).

// Where a lane's fragments start in an activation unit of T rows (8 or 1)
template <int T>
struct MmaUnit {
    static constexpr int kStretch = 64 * T;  // codes of a 64-element stretch
    static constexpr int kBlock = 4 * T;     // 32-element formats: from a block's scales to the next block's
    static constexpr int kStart = (kImgStart - kImgD) * T;  // from a scale to the accumulator start
    int bytes;       // of a unit
    int code, sums;  // this lane's 16 bytes of a stretch, its 8 bytes of sums
    int col;         // this lane's first column (4 bytes each); with one row both columns are that row
    __device__ __forceinline__ MmaUnit(int unit_bytes, int lane) : bytes(unit_bytes) {
        const int row = T == 8 ? lane >> 2 : 0, tig = lane & 3;
        code = (row * 4 + tig) * 16;
        sums = kImgSums * T + (row * 4 + tig) * 8;
        col = T == 8 ? tig * 8 : 0;
    }
    __device__ __forceinline__ uint2 columns(const uint8_t *p) const {
        if (T == 8) return *reinterpret_cast<const uint2 *>(p + col);
        const uint32_t v = *reinterpret_cast<const uint32_t *>(p);
        return make_uint2(v, v);
    }
    __device__ __forceinline__ float2 scales(const uint8_t *p) const {
        const uint2 v = columns(p);
        return make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
    }
};

__device__ __forceinline__ uint32_t lds32(const uint8_t *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ float lds_f16(const uint8_t *p) { return f16_bits_to_f32(*reinterpret_cast<const unsigned short *>(p)); }

template <bool FIVE_BIT>
struct MmaQ4or5K {
    static constexpr int kBytes = FIVE_BIT ? Q5K_BYTES : Q4K_BYTES;
    static constexpr int kKind = kImgK, kOffset = 0;  // order of the activation codes, code offset of the weights
    static constexpr bool kTwoSums = true;            // the instances with two sums per warp exist (two_sums, lloom_b200.cu)
    template <int NT, int T>
    __device__ static __forceinline__ void superblock(const uint8_t *ra, const uint8_t *rb, const uint8_t *act, const MmaUnit<T> &u, int lane, int,
                                                      float (&out)[NT][4]) {
        const int tig = lane & 3;
        const uint4 ha = *reinterpret_cast<const uint4 *>(ra), hb = *reinterpret_cast<const uint4 *>(rb);
        // 6-bit scales / mins (utils.rs:50-60), four per word, for the two rows
        const uint32_t sca[2] = {ha.y & 0x3f3f3f3fu, (ha.w & 0x0f0f0f0fu) | (((ha.y >> 6) & 0x03030303u) << 4)};
        const uint32_t scb[2] = {hb.y & 0x3f3f3f3fu, (hb.w & 0x0f0f0f0fu) | (((hb.y >> 6) & 0x03030303u) << 4)};
        const uint32_t mna[2] = {ha.z & 0x3f3f3f3fu, ((ha.w >> 4) & 0x0f0f0f0fu) | (((ha.z >> 6) & 0x03030303u) << 4)};
        const uint32_t mnb[2] = {hb.z & 0x3f3f3f3fu, ((hb.w >> 4) & 0x0f0f0f0fu) | (((hb.z >> 6) & 0x03030303u) << 4)};
        uint2 qha = make_uint2(0, 0), qhb = make_uint2(0, 0);
        if (FIVE_BIT) {  // fifth bits of bytes 8tig .. 8tig + 7, bit j = sub-block j
            qha = *reinterpret_cast<const uint2 *>(ra + 16 + 8 * tig);
            qhb = *reinterpret_cast<const uint2 *>(rb + 16 + 8 * tig);
        }
        const uint8_t *qa = ra + (FIVE_BIT ? 48 : 16) + 8 * tig, *qb = rb + (FIVE_BIT ? 48 : 16) + 8 * tig;
        int S[NT][4], Sh[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) S[nt][i] = Sh[nt][i] = 0;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const uint2 wa = *reinterpret_cast<const uint2 *>(qa + 32 * g), wb = *reinterpret_cast<const uint2 *>(qb + 32 * g);
            uint32_t alo[4] = {wa.x & 0x0f0f0f0fu, wb.x & 0x0f0f0f0fu, wa.y & 0x0f0f0f0fu, wb.y & 0x0f0f0f0fu};
            // Q4_K: high nibbles stay in place (16 q, unsigned bytes); the factor 16 comes out of the sum, exactly
            uint32_t ahi[4] = {wa.x & 0xf0f0f0f0u, wb.x & 0xf0f0f0f0u, wa.y & 0xf0f0f0f0u, wb.y & 0xf0f0f0f0u};
            if (FIVE_BIT) {
#pragma unroll
                for (int i = 0; i < 4; ++i) ahi[i] >>= 4;
                const uint32_t h[4] = {qha.x, qhb.x, qha.y, qhb.y};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    alo[i] |= ((h[i] >> (2 * g)) & 0x01010101u) << 4;
                    ahi[i] |= ((h[i] >> (2 * g + 1)) & 0x01010101u) << 4;
                }
            }
            const int sel = 0x4440 + 2 * (g & 1);  // byte of the scale word, zero-extended
            const int sa_lo = __byte_perm(sca[g >> 1], 0, sel), sa_hi = __byte_perm(sca[g >> 1], 0, sel + 1);
            const int sb_lo = __byte_perm(scb[g >> 1], 0, sel), sb_hi = __byte_perm(scb[g >> 1], 0, sel + 1);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint4 bv = *reinterpret_cast<const uint4 *>(act + nt * u.bytes + g * MmaUnit<T>::kStretch + u.code);
                int cl[4] = {0, 0, 0, 0}, ch[4] = {0, 0, 0, 0};
                mma_s8_k32(cl, alo, bv.x, bv.y);
                S[nt][0] += sa_lo * cl[0];
                S[nt][1] += sa_lo * cl[1];
                S[nt][2] += sb_lo * cl[2];
                S[nt][3] += sb_lo * cl[3];
                int(&H)[4] = FIVE_BIT ? S[nt] : Sh[nt];
                if (FIVE_BIT) mma_s8_k32(ch, ahi, bv.z, bv.w);
                else mma_u8_k32(ch, ahi, bv.z, bv.w);
                H[0] += sa_hi * ch[0];
                H[1] += sa_hi * ch[1];
                H[2] += sb_hi * ch[2];
                H[3] += sb_hi * ch[3];
            }
        }
        // min term: A[row][2j], A[row][2j + 1] = m_j against the two 16-element sums of sub-block j, all exact in f16
        const uint32_t sel = 0x4040u + 0x0101u * (uint32_t)tig;  // bytes m, 0x64, m, 0x64: the f16 pair 1024 + m
        uint32_t am[4] = {__byte_perm(mna[0], 0x64u, sel), __byte_perm(mnb[0], 0x64u, sel), __byte_perm(mna[1], 0x64u, sel),
                          __byte_perm(mnb[1], 0x64u, sel)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&am[i]), __float2half2_rn(1024.0f));
            am[i] = *reinterpret_cast<const uint32_t *>(&h);
        }
        const float dwa = f16_bits_to_f32(ha.x & 0xffffu), dma = f16_bits_to_f32(ha.x >> 16);
        const float dwb = f16_bits_to_f32(hb.x & 0xffffu), dmb = f16_bits_to_f32(hb.x >> 16);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
            for (int i = 0; i < 4; ++i) S[nt][i] += Sh[nt][i] >> 4;
            const uint2 bm = *reinterpret_cast<const uint2 *>(act + nt * u.bytes + u.sums);
            float mn[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16_k16(mn, am, bm.x, bm.y);
            const float2 da = u.scales(act + nt * u.bytes + kImgKD * T);
            auto term = [](float da, float dw, float dm, int s, float mn) {
                return fmaf(__fmul_rn(-da, dm), mn, __fmul_rn(__fmul_rn(da, dw), (float)s));
            };
            out[nt][0] = __fadd_rn(out[nt][0], term(da.x, dwa, dma, S[nt][0], mn[0]));
            out[nt][1] = __fadd_rn(out[nt][1], term(da.y, dwa, dma, S[nt][1], mn[1]));
            out[nt][2] = __fadd_rn(out[nt][2], term(da.x, dwb, dmb, S[nt][2], mn[2]));
            out[nt][3] = __fadd_rn(out[nt][3], term(da.y, dwb, dmb, S[nt][3], mn[3]));
        }
    }
};
struct MmaQ4K : MmaQ4or5K<false> {};
struct MmaQ5K : MmaQ4or5K<true> {};

struct MmaQ6K {
    static constexpr int kBytes = Q6K_BYTES;
    static constexpr int kKind = kImgQ6K, kOffset = 0;
    static constexpr bool kTwoSums = false;
    template <int NT, int T>
    __device__ static __forceinline__ void superblock(const uint8_t *ra, const uint8_t *rb, const uint8_t *act, const MmaUnit<T> &u, int lane, int,
                                                      float (&out)[NT][4]) {
        const int tig = lane & 3;
        // 210-byte superblocks: 2-byte aligned, read as aligned words and shifted together
        const uint32_t sha = (smem_u32(ra) & 2u) * 8u, shb = (smem_u32(rb) & 2u) * 8u;
        const uint8_t *wa = ra - (sha >> 3), *wb = rb - (shb >> 3);
        uint32_t sca[4], scb[4];  // the sixteen signed scales
        {
            uint32_t pa = lds32(wa + 192), pb = lds32(wb + 192);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t na = lds32(wa + 196 + 4 * i), nb = lds32(wb + 196 + 4 * i);
                sca[i] = __funnelshift_r(pa, na, sha);
                scb[i] = __funnelshift_r(pb, nb, shb);
                pa = na;
                pb = nb;
            }
        }
        auto word = [](const uint8_t *w, int off, uint32_t sh) { return __funnelshift_r(lds32(w + off), lds32(w + off + 4), sh); };
        int S[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) S[nt][i] = 0;
#pragma unroll
        for (int hs = 0; hs < 4; ++hs) {
            const int h = hs >> 1, s = hs & 1;
            const int lo = 64 * h + 16 * s + 4 * tig, hi = 128 + 32 * h + 16 * s + 4 * tig;
            uint32_t a[4], b[4];  // rows gid / gid + 8: code words of the sub-blocks gq = 0..3
            auto codes = [&](const uint8_t *w, uint32_t sh, uint32_t (&c)[4]) {
                const uint32_t la = word(w, lo, sh), lb = word(w, lo + 32, sh), hh = word(w, hi, sh);
                c[0] = (la & 0x0f0f0f0fu) | ((hh << 4) & 0x30303030u);
                c[1] = (lb & 0x0f0f0f0fu) | ((hh << 2) & 0x30303030u);
                c[2] = ((la >> 4) & 0x0f0f0f0fu) | (hh & 0x30303030u);
                c[3] = ((lb >> 4) & 0x0f0f0f0fu) | ((hh >> 2) & 0x30303030u);
#pragma unroll
                for (int i = 0; i < 4; ++i) c[i] = (c[i] + 0x60606060u) ^ 0x80808080u;  // code - 32 per byte: no carry leaves a byte
            };
            codes(wa, sha, a);
            codes(wb, shb, b);
            int sa[4], sb[4];
#pragma unroll
            for (int gq = 0; gq < 4; ++gq) {  // scale 8h + s + 2gq
                const int idx = 8 * h + s + 2 * gq;
                sa[gq] = (int)(int8_t)(sca[idx >> 2] >> (8 * (idx & 3)));
                sb[gq] = (int)(int8_t)(scb[idx >> 2] >> (8 * (idx & 3)));
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint4 bv = *reinterpret_cast<const uint4 *>(act + nt * u.bytes + hs * MmaUnit<T>::kStretch + u.code);
                const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                for (int gq = 0; gq < 4; ++gq) {
                    int c[4] = {0, 0, 0, 0};
                    mma_s8_k16(c, a[gq], b[gq], bw[gq]);
                    S[nt][0] += sa[gq] * c[0];
                    S[nt][1] += sa[gq] * c[1];
                    S[nt][2] += sb[gq] * c[2];
                    S[nt][3] += sb[gq] * c[3];
                }
            }
        }
        const float dwa = lds_f16(ra + 208), dwb = lds_f16(rb + 208);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const float2 da = u.scales(act + nt * u.bytes + kImgKD * T);
            out[nt][0] = __fadd_rn(out[nt][0], __fmul_rn(__fmul_rn(da.x, dwa), (float)S[nt][0]));
            out[nt][1] = __fadd_rn(out[nt][1], __fmul_rn(__fmul_rn(da.y, dwa), (float)S[nt][1]));
            out[nt][2] = __fadd_rn(out[nt][2], __fmul_rn(__fmul_rn(da.x, dwb), (float)S[nt][2]));
            out[nt][3] = __fadd_rn(out[nt][3], __fmul_rn(__fmul_rn(da.y, dwb), (float)S[nt][3]));
        }
    }
};

// The 32-element formats, two blocks at a time: rows are multiples of 64 elements, so a pair of blocks starts on a 4-byte
// boundary and the first block's codes lie 2 bytes past one, the second's on one.
enum { kFmtQ8_0, kFmtQ4_0, kFmtQ5_0 };
template <int FMT>
struct MmaBlocks32 {
    static constexpr int kBlk = FMT == kFmtQ8_0 ? Q8_0_BYTES : FMT == kFmtQ4_0 ? Q4_0_BYTES : Q5_0_BYTES;
    static constexpr int kBytes = 8 * kBlk;
    static constexpr int kKind = FMT == kFmtQ8_0 ? kImg32 : kImgSplit, kOffset = FMT == kFmtQ8_0 ? 0 : FMT == kFmtQ4_0 ? 8 : 16;
    static constexpr bool kTwoSums = false;
    // A fragments (k = 4tig.., 16 + 4tig.. as the image orders the codes) and scale of the even / odd block of a pair
    __device__ static __forceinline__ void pair(const uint8_t *p, int tig, uint32_t (&even)[2], uint32_t (&odd)[2], float &d_even,
                                                float &d_odd) {
        if (FMT == kFmtQ8_0) {
            const uint8_t *q = p + 8 * tig;
            const uint32_t w0 = lds32(q), w1 = lds32(q + 4), w2 = lds32(q + 8);
            even[0] = __funnelshift_r(w0, w1, 16);
            even[1] = __funnelshift_r(w1, w2, 16);
            odd[0] = lds32(q + 36);
            odd[1] = lds32(q + 40);
            d_even = lds_f16(p);
            d_odd = lds_f16(p + 34);
        } else if (FMT == kFmtQ4_0) {
            const uint8_t *q = p + 4 * tig;
            const uint32_t we = __funnelshift_r(lds32(q), lds32(q + 4), 16), wo = lds32(q + 20);
            even[0] = we & 0x0f0f0f0fu;
            even[1] = (we >> 4) & 0x0f0f0f0fu;
            odd[0] = wo & 0x0f0f0f0fu;
            odd[1] = (wo >> 4) & 0x0f0f0f0fu;
            d_even = lds_f16(p);
            d_odd = lds_f16(p + 18);
        } else {
            const uint8_t *q = p + 4 * tig;
            const uint32_t h0 = lds32(p), h1 = lds32(p + 4);
            const uint32_t bits_e = __funnelshift_r(h0, h1, 16), bits_o = lds32(p + 24);
            const uint32_t we = __funnelshift_r(lds32(q + 4), lds32(q + 8), 16), wo = lds32(q + 28);
            auto spread = [](uint32_t b) { return ((b & 0xFu) * 0x00204081u & 0x01010101u) << 4; };  // four bits to four bytes
            even[0] = (we & 0x0f0f0f0fu) | spread(bits_e >> (4 * tig));
            even[1] = ((we >> 4) & 0x0f0f0f0fu) | spread(bits_e >> (16 + 4 * tig));
            odd[0] = (wo & 0x0f0f0f0fu) | spread(bits_o >> (4 * tig));
            odd[1] = ((wo >> 4) & 0x0f0f0f0fu) | spread(bits_o >> (16 + 4 * tig));
            d_even = f16_bits_to_f32(h0 & 0xffffu);
            d_odd = lds_f16(p + 22);
        }
    }
    template <int NT, int T>
    __device__ static __forceinline__ void superblock(const uint8_t *ra, const uint8_t *rb, const uint8_t *act, const MmaUnit<T> &u, int lane, int nblk,
                                                      float (&out)[NT][4]) {
        const int tig = lane & 3;
        float low[NT][4], high[NT][4];  // block pairs (0 + 1) and (2 + 3) of the superblock
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            if (2 * g >= nblk) {  // warp-uniform: the end of a row that is not a whole number of 256-element spans
                if (g == 1 || g == 2) {
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int i = 0; i < 4; ++i) high[nt][i] = 0.0f;
                }
                break;
            }
            uint32_t ae[2], ao[2], be[2], bo[2];
            float dae, dao, dbe, dbo;
            pair(ra + 2 * kBlk * g, tig, ae, ao, dae, dao);
            pair(rb + 2 * kBlk * g, tig, be, bo, dbe, dbo);
            const uint32_t fe[4] = {ae[0], be[0], ae[1], be[1]}, fo[4] = {ao[0], bo[0], ao[1], bo[1]};
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint8_t *a = act + nt * u.bytes;
                const uint4 bv = *reinterpret_cast<const uint4 *>(a + g * MmaUnit<T>::kStretch + u.code);
                const uint8_t *d = a + kImgD * T + 2 * g * u.kBlock;
                uint2 se = make_uint2(kMagicBits, kMagicBits), so = se;
                if (FMT != kFmtQ8_0) {
                    se = u.columns(d + u.kStart);
                    so = u.columns(d + u.kStart + u.kBlock);
                }
                int c[4];
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                mma_s8_k32_from(c, fe, bv.x, bv.y, (int)se.x, (int)se.y);
                add(v, c, u.scales(d), dae, dbe);
                mma_s8_k32_from(c, fo, bv.z, bv.w, (int)so.x, (int)so.y);
                add(v, c, u.scales(d + u.kBlock), dao, dbo);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (g == 0) low[nt][i] = v[i];
                    if (g == 1) low[nt][i] = __fadd_rn(low[nt][i], v[i]);
                    if (g == 2) high[nt][i] = v[i];
                    if (g == 3) high[nt][i] = __fadd_rn(high[nt][i], v[i]);
                }
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) out[nt][i] = __fadd_rn(out[nt][i], __fadd_rn(low[nt][i], high[nt][i]));
    }
    // Q8_0 / Q4_0: out += (d_w * d_a) * dot, the AVX2 arm's product and fused multiply-add; Q5_0: ((dot * d_w) * d_a), the
    // scalar arm's (the only one it has)
    __device__ static __forceinline__ void add(float (&out)[4], const int (&c)[4], float2 da, float dwa, float dwb) {
        const float v0 = __int_as_float(c[0]) - kMagic, v1 = __int_as_float(c[1]) - kMagic;
        const float v2 = __int_as_float(c[2]) - kMagic, v3 = __int_as_float(c[3]) - kMagic;
        if (FMT == kFmtQ5_0) {
            out[0] = __fadd_rn(out[0], __fmul_rn(__fmul_rn(v0, dwa), da.x));
            out[1] = __fadd_rn(out[1], __fmul_rn(__fmul_rn(v1, dwa), da.y));
            out[2] = __fadd_rn(out[2], __fmul_rn(__fmul_rn(v2, dwb), da.x));
            out[3] = __fadd_rn(out[3], __fmul_rn(__fmul_rn(v3, dwb), da.y));
        } else {
            out[0] = fmaf(__fmul_rn(dwa, da.x), v0, out[0]);
            out[1] = fmaf(__fmul_rn(dwa, da.y), v1, out[1]);
            out[2] = fmaf(__fmul_rn(dwb, da.x), v2, out[2]);
            out[3] = fmaf(__fmul_rn(dwb, da.y), v3, out[3]);
        }
    }
};
struct MmaQ8_0 : MmaBlocks32<kFmtQ8_0> {};
struct MmaQ4_0 : MmaBlocks32<kFmtQ4_0> {};
struct MmaQ5_0 : MmaBlocks32<kFmtQ5_0> {};

// ---- the kernel ----

// Producer warp.  Stages in order, tile group by tile group, slice by slice along the row: `slice_sb` superblocks of up to TR
// tiles of 16 rows and, when the activations are streamed, the same superblocks of the image (one bulk copy).  The
// activations are the stream predecessor's work: the first stages' weights are requested before it has finished, their
// activations after.
//
// Weights: where rows are multiples of 16 bytes, one or two tiled TMA loads per 16-row tile (boxes of 16 rows x `row_pitch`
// bytes of one or half a slice: the padding that keeps rows on distinct banks is simply more of the row, 16 to 32 bytes).
// A bulk copy per row costs its SM 29 ns plus 9 ns per KB whatever issues it -- 4.2 TB/s on 148 SMs at 1 KB, 6.5 from 2 KB
// up, where boxes reach 6.6 to 7.0 -- so other row lengths, whose rows start anywhere, are copied in long slices.
// One warp on a scheduler that sixteen computing warps keep busy: with divisions and 64-bit products per stage its own
// instructions took 2 us for each, so they are kept few.
__device__ __forceinline__ void tma_box(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mma_producer(const GemvParams &p, const CUtensorMap *map, uint64_t *full, uint64_t *empty, uint8_t *stage0,
                                             int r_begin, int r_end, int lane, const uint8_t *img, int nt_g) {
    const int nsb = p.nsb, slice_sb = p.slice_sb, stages = p.stages;
    const uint32_t unit_row = (uint32_t)(nt_g * p.img_unit);
    const uint32_t row_bytes = (uint32_t)p.row_bytes, slice = (uint32_t)p.slice_bytes;
    const int64_t bulk_limit = p.w_bytes & ~(int64_t)15;  // bytes the bulk engine may touch
    int issued = 0;           // stages requested so far
    bool acts_ready = false;  // the stream predecessor has finished
    auto send_acts = [&](int s, int sb0) {
        const uint32_t bytes = (uint32_t)min(slice_sb, nsb - sb0) * unit_row;
        bulk_g2s(stage0 + (size_t)s * p.stage_bytes + p.act_stage_off, img + (size_t)sb0 * unit_row, bytes, &full[s]);
    };
    auto first_acts = [&]() {  // the activations of the stages requested so far
        asm volatile("griddepcontrol.wait;" ::: "memory");
        acts_ready = true;
        if (lane == 0)
            for (int j = 0, sb0 = 0; j < issued; ++j) {
                send_acts(j, sb0);
                sb0 = sb0 + slice_sb < nsb ? sb0 + slice_sb : 0;
            }
    };
    int s = 0;
    uint32_t phase = 1;  // parity of the empty barrier's phase before the one that frees the stage
    for (int row0 = r_begin; row0 < r_end; row0 += p.tile_rows_cta) {
        const int rows = min(p.tile_rows_cta, r_end - row0);
        const int64_t base = (int64_t)row0 * row_bytes;
        uint32_t at = 0;  // bytes into a row
        for (int sb0 = 0; sb0 < nsb; sb0 += slice_sb, at += slice) {
            if (issued == stages && p.act_stream && !acts_ready) first_acts();
            if (issued >= stages && !mbar_wait(&empty[s], phase)) return;
            uint8_t *dst = stage0 + (size_t)s * p.stage_bytes;
            const uint32_t act = p.act_stream ? (uint32_t)min(slice_sb, nsb - sb0) * unit_row : 0u;
            if (p.boxes) {
                if (lane == 0) {
                    const int tiles = (rows + kMmaTileRows - 1) / kMmaTileRows;
                    mbar_arrive_expect_tx(&full[s], (uint32_t)(tiles * p.boxes * p.box_bytes) + act);  // rows and bytes past the end count
                    int x = (int)(at >> 4) * 2;  // in elements of 8 bytes, on a 16-byte boundary
                    for (int b = 0; b < p.boxes; ++b, x += p.box_step)
                        for (int t = 0; t < tiles; ++t)
                            tma_box(dst + (t * p.boxes + b) * p.box_bytes, map, x, row0 + t * kMmaTileRows, &full[s]);
                }
            } else {
                const uint32_t len = min(slice, row_bytes - at);
                uint32_t bytes = 0;
                for (int r = lane; r < rows; r += 32) {
                    const int64_t start = base + (int64_t)r * row_bytes + at, end = start + len, a0 = start & ~(int64_t)15;
                    const int64_t a1 = min((end + 15) & ~(int64_t)15, bulk_limit);
                    if (a1 > a0) bytes += (uint32_t)(a1 - a0);
                    // ragged end of the matrix: plain loads
                    for (int64_t i = a1 > a0 ? a1 : a0; i < end; ++i) dst[r * p.row_pitch + (i - a0)] = __ldg(p.w + i);
                }
                bytes = __reduce_add_sync(0xffffffffu, bytes);
                __syncwarp();
                if (lane == 0) mbar_arrive_expect_tx(&full[s], bytes + act);
                __syncwarp();
                for (int r = lane; r < rows; r += 32) {
                    const int64_t start = base + (int64_t)r * row_bytes + at, end = start + len, a0 = start & ~(int64_t)15;
                    const int64_t a1 = min((end + 15) & ~(int64_t)15, bulk_limit);
                    if (a1 > a0) bulk_g2s(dst + r * p.row_pitch, p.w + a0, (uint32_t)(a1 - a0), &full[s]);
                }
            }
            if (acts_ready && p.act_stream && lane == 0) send_acts(s, sb0);
            __syncwarp();
            ++issued;
            if (++s == stages) {
                s = 0;
                phase ^= 1;
            }
        }
    }
    if (p.act_stream && !acts_ready) first_acts();  // the whole range fits the ring
}

// Dynamic shared memory: [barriers 128 B][partial sums][resident activations][staged output rows, fused gather only][stages]
// SUMS = 2: a warp keeps the sums of two slots, j and j + S, in turn (S = 4, slices of eight superblocks).
// EPI = 1: the instance with the store blocks and the fused gather (up to eight rows).
template <class Fmt, int NT, int T, int SUMS, int EPI>
__global__ void __launch_bounds__(32 * (kMmaWarps + 1), 1) gemv_mma_kernel(const GemvParams p, const __grid_constant__ CUtensorMap map) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + kMmaStages;
    uint64_t *act_bar = empty + kMmaStages;
    int *cta_ok = reinterpret_cast<int *>(smem + kMmaBarBytes - 8);  // cleared by a warp whose bounded wait ran out
    float4 *red = reinterpret_cast<float4 *>(smem + kMmaBarBytes);
    uint8_t *act_res = smem + kMmaBarBytes + p.red_bytes;
    float *out_s = reinterpret_cast<float *>(act_res + p.act_bytes);
    uint8_t *stage0 = act_res + p.act_bytes + p.out_bytes;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total_tiles = (p.n + kMmaTileRows - 1) / kMmaTileRows;
    const int r_begin = (int)(((int64_t)blockIdx.x * total_tiles) / gridDim.x) * kMmaTileRows;
    const int r_end = min(p.n, (int)(((int64_t)(blockIdx.x + 1) * total_tiles) / gridDim.x) * kMmaTileRows);
    // this CTA's group of activation tiles (the image is padded to whole groups)
    const int nt_g = p.group_nt, tile0 = blockIdx.y * nt_g;
    const uint8_t *img = p.img + (int64_t)tile0 * p.nsb * p.img_unit;

    if (threadIdx.x < p.stages) {
        mbar_init(&full[threadIdx.x], 1);
        mbar_init(&empty[threadIdx.x], p.n_cwarps);
    }
    if (threadIdx.x == 32) mbar_init(act_bar, 1);
    if (threadIdx.x == 0) *cta_ok = 1;
    fence_mbar_init();
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == p.n_cwarps) {
        mma_producer(p, &map, full, empty, stage0, r_begin, r_end, lane, img, nt_g);
        return;
    }

    const int nthreads = p.n_cwarps * 32;
    bool alive = true;  // after a timed-out wait the warp keeps meeting its team at the barriers but computes nothing
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (EPI != 0 && p.wait_flags) alive = wait_exchange(p);  // x came out of a fused gather: all peers' rows are in
    if (!p.act_stream) {
        if (p.x) {  // quantizer as prologue: a warp's blocks are loaded four at a time, one L2 round trip per batch
            const int nblk = p.m * p.nsb;
            for (int base = warp; base < nblk; base += 4 * p.n_cwarps) {
                float v[4][8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int blk = base + j * p.n_cwarps, t = blk / p.nsb, e0 = (blk - t * p.nsb) * 256 + lane * 8;
                    const bool live = blk < nblk && e0 < p.k;
                    if (live) load8(p.x, p.x_type, (int64_t)t * p.k + e0, v[j]);
                    else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[j][i] = 0.0f;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int blk = base + j * p.n_cwarps, t = blk / p.nsb, sb = blk - t * p.nsb;
                    if (blk < nblk)
                        values_to_image(v[j], act_res + (size_t)sb * p.img_unit, Fmt::kKind, Fmt::kOffset, T, t, lane, sb * 256 + lane * 8 < p.k);
                }
            }
            asm volatile("bar.sync 15, %0;" ::"r"(nthreads) : "memory");
        } else if (p.img) {
            if (threadIdx.x == 0) {
                mbar_arrive_expect_tx(act_bar, (uint32_t)p.act_copy);
                bulk_g2s(act_res, img, (uint32_t)p.act_copy, act_bar);
            }
            alive = mbar_wait(act_bar, 0) && alive;
        } else {
            blocks_to_image(p.act, act_res, Fmt::kKind, Fmt::kOffset, p.img_unit, p.m, p.k, 1, T, threadIdx.x, nthreads);
            asm volatile("bar.sync 15, %0;" ::"r"(nthreads) : "memory");
        }
    }

    const int S = p.split, slot = warp % S, team = warp / S;
    const int tn = team % p.col_parts, tr = team / p.col_parts;
    const int gid = lane >> 2, tig = lane & 3;
    // column part: NT activation tiles from nt0 on; parts overlap where the tiles do not divide (the same values twice)
    const int nt0 = min(tn * NT, nt_g - NT);
    const int nt_skip = tn * NT - nt0;  // tiles of this part that the part before it stores
    const int unit_row = nt_g * p.img_unit;
    const MmaUnit<T> unit(p.img_unit, lane);
    const GemvSeg sg = gemv_segment<false>(p, 0, r_begin, r_end);
    const int sl_step = p.slice_bytes & 15;
    int s = 0;
    uint32_t phase = 0;
    for (int g0 = r_begin; g0 < r_end; g0 += p.tile_rows_cta) {
        const int trow = g0 + tr * kMmaTileRows;
        const int rows = min(kMmaTileRows, r_end - trow);  // <= 0: this warp has no tile in the group
        // rows past the end of the range read row 0 of the tile and are dropped later
        const int la = tr * kMmaTileRows + (gid < rows ? gid : 0), lb = tr * kMmaTileRows + (gid + 8 < rows ? gid + 8 : 0);
        // where the rows' slices start within their 16-byte lines (changes from slice to slice by a constant)
        int offa = (int)((uint32_t)(g0 + la) * (uint32_t)p.row_bytes & 15u), offb = (int)((uint32_t)(g0 + lb) * (uint32_t)p.row_bytes & 15u);
        const uint8_t *rowa, *rowb;  // this slot's first superblock of the two rows, in stage 0
        if (p.boxes) {
            const int box = slot >= p.box_sb ? 1 : 0;
            const uint8_t *tile = stage0 + (tr * p.boxes + box) * p.box_bytes + (slot - box * p.box_sb) * Fmt::kBytes;
            rowa = tile + (la - tr * kMmaTileRows) * p.row_pitch;
            rowb = tile + (lb - tr * kMmaTileRows) * p.row_pitch;
        } else {
            rowa = stage0 + la * p.row_pitch + slot * Fmt::kBytes;
            rowb = stage0 + lb * p.row_pitch + slot * Fmt::kBytes;
        }
        float out[NT][4], other[NT][4];  // other: the second slot's sums
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) out[nt][i] = other[nt][i] = 0.0f;
        for (int sb0 = 0; sb0 < p.nsb; sb0 += p.slice_sb) {
            alive = alive && mbar_wait(&full[s], phase);
            const int st = s * p.stage_bytes, n_sb = alive && rows > 0 ? min(p.slice_sb, p.nsb - sb0) : 0;
            auto work = [&](int j, int ahead, float(&sum)[NT][4]) {
                const uint8_t *act = (p.act_stream ? stage0 + st + p.act_stage_off + j * unit_row : act_res + (sb0 + j) * unit_row) + nt0 * p.img_unit;
                const int nblk = min(8, (p.k >> 5) - (sb0 + j) * 8);
                Fmt::template superblock<NT, T>(rowa + st + offa + ahead, rowb + st + offb + ahead, act, unit, lane, nblk, sum);
            };
            if (SUMS == 2) {
                if (slot < n_sb) work(slot, 0, out);
                if (slot + S < n_sb) work(slot + S, p.second, other);
            } else {
                for (int j = slot; j < n_sb; j += S) work(j, (j - slot) * Fmt::kBytes, out);
            }
            offa = (offa + sl_step) & 15;
            offb = (offb + sl_step) & 15;
            // this warp is done reading the stage once the sums its loads feed have been computed
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    pin_value(out[nt][i]);
                    if (SUMS == 2) pin_value(other[nt][i]);
                }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (++s == p.stages) {
                s = 0;
                phase ^= 1;
            }
        }
        if (SUMS == 2) {  // slots j and j + 4: the first step of add_slots
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i) out[nt][i] = __fadd_rn(out[nt][i], other[nt][i]);
        }
        // partial sums of the team meet in shared memory; its first warp adds them
        if (S > 1) {
            float4 *part = red + (size_t)team * (S - 1) * NT * 32 + lane;
            if (slot != 0) {
                if (g0 != r_begin) asm volatile("bar.sync %0, %1;" ::"r"(2 + 2 * team), "r"(S * 32) : "memory");  // the last group's have been read
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    part[((slot - 1) * NT + nt) * 32] = make_float4(out[nt][0], out[nt][1], out[nt][2], out[nt][3]);
                asm volatile("bar.arrive %0, %1;" ::"r"(1 + 2 * team), "r"(S * 32) : "memory");
                continue;
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + 2 * team), "r"(S * 32) : "memory");
            auto plus = [](float4 a, float4 b) {
                return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
            };
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {  // the order of add_slots
                auto at = [&](int j) { return part[((j - 1) * NT + nt) * 32]; };
                float4 v = make_float4(out[nt][0], out[nt][1], out[nt][2], out[nt][3]);
                if (S == 8) v = plus(plus(plus(v, at(4)), plus(at(2), at(6))), plus(plus(at(1), at(5)), plus(at(3), at(7))));
                else if (S == 4) v = plus(plus(v, at(2)), plus(at(1), at(3)));
                else v = plus(v, at(1));
                out[nt][0] = v.x;
                out[nt][1] = v.y;
                out[nt][2] = v.z;
                out[nt][3] = v.w;
            }
            if (g0 + p.tile_rows_cta < r_end) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) pin_value(out[nt][i]);
                asm volatile("bar.arrive %0, %1;" ::"r"(2 + 2 * team), "r"(S * 32) : "memory");
            }
        }
        if (!alive) continue;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            if (nt < nt_skip) continue;
            const int t = (tile0 + nt0 + nt) * 8 + 2 * tig;  // activation rows of this lane's columns
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = gid + 8 * (i >> 1), c = t + (i & 1);
                if (r < rows && c < p.m) {
                    if (EPI == 0) store_y(p.y, p.y_type, (int64_t)c * p.ldy + trow + r, out[nt][i]);
                    else emit_out(p, sg, out_s, c, trow + r, out[nt][i]);
                }
            }
        }
    }
    if (EPI != 0 && (p.out_bytes || p.publish)) {  // every consumer warp gets here, timed-out ones included
        if (!alive) *cta_ok = 0;
        asm volatile("bar.sync 15, %0;" ::"r"(nthreads) : "memory");
        // staged rows leave for the peers only if every warp finished its tiles (a timed-out warp left gaps)
        if (p.out_bytes && *cta_ok) flush_out(p, out_s, r_begin, r_end, threadIdx.x, nthreads);
        if (p.publish) {
            asm volatile("bar.sync 15, %0;" ::"r"(nthreads) : "memory");
            if (threadIdx.x == 0) publish_arrival(p);
        }
    }
}

// ---- launchers of one format ----

template <class Fmt, int NT, int T, int SUMS, int EPI>
static cudaError_t launch_mma_inst(const GemvParams &p, const CUtensorMap &map, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream) {
    auto kern = gemv_mma_kernel<Fmt, NT, T, SUMS, EPI>;
    static FuncSmemConfig cfg;
    cudaError_t e = ensure_smem(kern, cfg, smem, false);
    if (e != cudaSuccess) return e;
    return launch_early(kern, dim3((unsigned)grid_x, (unsigned)grid_y), 32 * (p.n_cwarps + 1), (size_t)smem, overlap, stream, p, map);
}

template <class Fmt, int T, int SUMS>
static cudaError_t launch_mma_tile(const GemvParams &p, const CUtensorMap &map, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream) {
    return gemv_needs_epi(p) ? launch_mma_inst<Fmt, 1, T, SUMS, 1>(p, map, grid_x, grid_y, smem, overlap, stream)
                             : launch_mma_inst<Fmt, 1, T, SUMS, 0>(p, map, grid_x, grid_y, smem, overlap, stream);
}

template <class Fmt>
static cudaError_t launch_mma_format(const GemvParams &p, const CUtensorMap &map, int nt, int grid_x, int grid_y, int smem, bool overlap, cudaStream_t stream) {
    if (p.second != 0) {  // two sums per warp
        if constexpr (Fmt::kTwoSums)
            if (nt == 1 && p.m > 1) return launch_mma_tile<Fmt, 8, 2>(p, map, grid_x, grid_y, smem, overlap, stream);
        return cudaErrorInvalidValue;
    }
    if (p.m == 1) return launch_mma_tile<Fmt, 1, 1>(p, map, grid_x, grid_y, smem, overlap, stream);
    if (nt == 1) return launch_mma_tile<Fmt, 8, 1>(p, map, grid_x, grid_y, smem, overlap, stream);
    if (gemv_needs_epi(p)) return cudaErrorInvalidValue;
    switch (nt) {
    case 2: return launch_mma_inst<Fmt, 2, 8, 1, 0>(p, map, grid_x, grid_y, smem, overlap, stream);
    case 3: return launch_mma_inst<Fmt, 3, 8, 1, 0>(p, map, grid_x, grid_y, smem, overlap, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace lloom
