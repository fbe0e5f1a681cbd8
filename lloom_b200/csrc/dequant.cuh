// Dequantize and row gather (embedding) for the six weight formats, exact T::to_float arithmetic.
//
// Bandwidth kernels (4 or 2 bytes out per element): one thread produces eight consecutive elements, two 16-byte stores,
// from loads as wide as the format's alignment allows.  With four elements per thread, byte loads, the format resolved at
// run time and a 64-bit division per thread, 512 rows of a 4096-wide Q6_K table took 5.6 us instead of 4.1.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace lloom {

// Eight bytes from a 2-byte aligned address
__device__ __forceinline__ uint2 ldg8_unaligned(const uint8_t *p) {
    const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
    return make_uint2((uint32_t)__ldg(h) | ((uint32_t)__ldg(h + 1) << 16), (uint32_t)__ldg(h + 2) | ((uint32_t)__ldg(h + 3) << 16));
}
__device__ __forceinline__ float ldg_f16(const uint8_t *p) { return f16_bits_to_f32(__ldg(reinterpret_cast<const unsigned short *>(p))); }

// Eight consecutive elements e .. e + 7 (e % 8 == 0) of a row of canonical blocks.
// Every product is an explicit round-to-nearest multiply: no contraction into FMA, so the values
// equal the reference's sequential f32 expressions bit for bit.
template <int DTYPE>
__device__ __forceinline__ void dequant8(const uint8_t *__restrict__ row, int64_t e, float (&r)[8]) {
    if (DTYPE == LLOOM_Q8_0) {
        // k_quants.rs:720-736   y = q as f32 * d
        const uint8_t *blk = row + (e >> 5) * Q8_0_BYTES;
        const float d = ldg_f16(blk);
        const uint2 q = ldg8_unaligned(blk + 2 + (e & 31));
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = __fmul_rn((float)(int8_t)((i < 4 ? q.x : q.y) >> (8 * (i & 3))), d);
    } else if (DTYPE == LLOOM_Q4_K || DTYPE == LLOOM_Q5_K) {
        // k_quants.rs:1747-1774   y = (d*sc)*q - (dmin*m); 2043-2076: the same with the fifth bit added to q in f32
        constexpr bool kFive = DTYPE == LLOOM_Q5_K;
        const uint8_t *blk = row + (e >> 8) * (kFive ? Q5K_BYTES : Q4K_BYTES);
        const int w = (int)(e & 255);
        const int g = w >> 6, hi = (w >> 5) & 1, t = w & 31;
        const uint4 head = __ldg(reinterpret_cast<const uint4 *>(blk));
        const float d = f16_bits_to_f32(head.x & 0xffffu), dmin = f16_bits_to_f32(head.x >> 16);
        const uint32_t s[3] = {head.y, head.z, head.w};
        int sc, mn;
        q4k_scale_min(s, 2 * g + hi, sc, mn);
        const float d1 = __fmul_rn(d, (float)sc), m1 = __fmul_rn(dmin, (float)mn);
        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(blk + (kFive ? 48 : 16) + 32 * g + t));
        uint2 h = make_uint2(0, 0);
        if (kFive) h = __ldg(reinterpret_cast<const uint2 *>(blk + 16 + t));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float v = (float)(((i < 4 ? q.x : q.y) >> (8 * (i & 3) + 4 * hi)) & 0xF);
            if (kFive) v = __fadd_rn(v, (((i < 4 ? h.x : h.y) >> (8 * (i & 3) + 2 * g + hi)) & 1u) ? 16.0f : 0.0f);
            r[i] = __fsub_rn(__fmul_rn(d1, v), m1);
        }
    } else if (DTYPE == LLOOM_Q4_0) {
        // k_quants.rs:299-318   y = (nibble - 8) as f32 * d; low nibbles are elements 0..15, high 16..31
        const uint8_t *blk = row + (e >> 5) * Q4_0_BYTES;
        const float d = ldg_f16(blk);
        const int w = (int)(e & 31), sh = (w & 16) ? 4 : 0;
        const uint2 q = ldg8_unaligned(blk + 2 + (w & 15));
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = __fmul_rn((float)((int)(((i < 4 ? q.x : q.y) >> (8 * (i & 3) + sh)) & 0xF) - 8), d);
    } else if (DTYPE == LLOOM_Q5_0) {
        // k_quants.rs:578-600   y = ((nibble | fifth bit << 4) - 16) as f32 * d
        const uint8_t *blk = row + (e >> 5) * Q5_0_BYTES;
        const float d = ldg_f16(blk);
        const unsigned short *h16 = reinterpret_cast<const unsigned short *>(blk + 2);
        const int w = (int)(e & 31), sh = (w & 16) ? 4 : 0;
        const uint32_t bits = ((uint32_t)__ldg(h16) | ((uint32_t)__ldg(h16 + 1) << 16)) >> w;
        const uint2 q = ldg8_unaligned(blk + 6 + (w & 15));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int nib = (int)(((i < 4 ? q.x : q.y) >> (8 * (i & 3) + sh)) & 0xF);
            r[i] = __fmul_rn((float)((nib | (int)(((bits >> i) & 1u) << 4)) - 16), d);
        }
    } else {
        // k_quants.rs:2327-2358   y = d * sc * q   (left to right)
        const uint8_t *blk = row + (e >> 8) * Q6K_BYTES;
        const int w = (int)(e & 255);
        const int h = w >> 7, gq = (w >> 5) & 3, l = w & 31;
        const float d = ldg_f16(blk + 208);
        const int sc = (int8_t)__ldg(blk + 192 + 8 * h + (l >> 4) + 2 * gq);
        const float dsc = __fmul_rn(d, (float)sc);
        const uint2 ql = ldg8_unaligned(blk + 64 * h + 32 * (gq & 1) + l), qh = ldg8_unaligned(blk + 128 + 32 * h + l);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t lo = ((i < 4 ? ql.x : ql.y) >> (8 * (i & 3) + ((gq & 2) ? 4 : 0))) & 0xF;
            const uint32_t hi = ((i < 4 ? qh.x : qh.y) >> (8 * (i & 3) + 2 * gq)) & 3;
            r[i] = __fmul_rn(dsc, (float)((int)(lo | (hi << 4)) - 32));
        }
    }
}

__device__ __forceinline__ void store8(float *out, const float (&r)[8]) {
    reinterpret_cast<float4 *>(out)[0] = make_float4(r[0], r[1], r[2], r[3]);
    reinterpret_cast<float4 *>(out)[1] = make_float4(r[4], r[5], r[6], r[7]);
}

template <int DTYPE, bool F16>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint8_t *__restrict__ blocks, int64_t elems, void *__restrict__ out) {
    const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (e >= elems) return;
    float r[8];
    dequant8<DTYPE>(blocks, e, r);
    if (F16) {
        __half2 h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(r[2 * i], r[2 * i + 1]);
        *reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(out) + e) = *reinterpret_cast<const uint4 *>(h);
    } else {
        store8(reinterpret_cast<float *>(out) + e, r);
    }
}

// out[i, :] = to_float(table row ids[i]); ids outside [0, rows) give a zero row.  blockIdx.x: id, blockIdx.y: part of a row.
template <int DTYPE>
__global__ void __launch_bounds__(256) get_rows_kernel(const uint8_t *__restrict__ blocks, int64_t rows, int64_t hidden, int64_t row_bytes,
                                                       const uint32_t *__restrict__ ids, int id_words, float *__restrict__ out) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t i = blockIdx.x, e = ((int64_t)blockIdx.y * blockDim.x + threadIdx.x) * 8;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (e >= hidden) return;
    const uint32_t id = __ldg(ids + i * id_words);
    float r[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if ((int64_t)id < rows) dequant8<DTYPE>(blocks + (int64_t)id * row_bytes, e, r);
    store8(out + i * hidden + e, r);
}

// f(format as a compile-time constant); the caller has checked that the format is one of the six
template <class F>
static void with_format(int dtype, F f) {
    switch (dtype) {
    case LLOOM_Q4_0: return f(std::integral_constant<int, LLOOM_Q4_0>());
    case LLOOM_Q5_0: return f(std::integral_constant<int, LLOOM_Q5_0>());
    case LLOOM_Q8_0: return f(std::integral_constant<int, LLOOM_Q8_0>());
    case LLOOM_Q4_K: return f(std::integral_constant<int, LLOOM_Q4_K>());
    case LLOOM_Q5_K: return f(std::integral_constant<int, LLOOM_Q5_K>());
    case LLOOM_Q6_K: return f(std::integral_constant<int, LLOOM_Q6_K>());
    }
}

}  // namespace lloom
