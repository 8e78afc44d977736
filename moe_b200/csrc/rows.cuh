// Activation rows: loads of f32 and bf16 rows, and the split forms that the expert kernels read.
#pragma once
#include "common.cuh"

namespace moexb {

// Position of input k inside a permuted activation row (see the header of stream.cuh).
__host__ __device__ constexpr int split_pos(int k) {
    const int G = k >> 6, kl = k & 63, t = kl >> 4, w = (kl >> 3) & 1, e = kl & 7;
    return G * 64 + w * 32 + t * 8 + (((e & 3) << 1) | (e >> 2));
}

// hi + lo halves of v as 16-bit patterns: fp16 (22 significand bits together) or bf16 (16 bits, full fp32 range)
template <bool F16>
__device__ __forceinline__ void split_hi_lo(float v, uint16_t& hi, uint16_t& lo) {
    if constexpr (F16) {
        const __half h = __float2half_rn(v), l = __float2half_rn(v - __half2float(h));
        hi = __half_as_ushort(h); lo = __half_as_ushort(l);
    } else {
        const __nv_bfloat16 h = __float2bfloat16_rn(v), l = __float2bfloat16_rn(v - __bfloat162float(h));
        hi = __bfloat16_as_ushort(h); lo = __bfloat16_as_ushort(l);
    }
}

// Place of input k in an activation row of the grouped GEMM (grouped.cuh).
template <bool Z>
__host__ __device__ constexpr int kslot(int k) {
    const int kk = k & 63, i = kk & 3, h = (kk >> 2) & 1, wd = kk >> 3;   // wd: the word of 8 nibbles
    const int t = Z ? ((wd >> 1) & 1) | ((wd & 1) << 1) : wd >> 1, hi = Z ? wd >> 2 : wd & 1;
    return (k & ~63) + 32 * hi + 16 * (i >> 1) + 4 * t + 2 * (i & 1) + h;
}
// Forms of a split activation row: 16-bit hi and lo halves in the order of split_pos (streaming kernels; fp16 or bf16) or of kslot
// (grouped GEMM; symmetric formats fp16, zero point bf16).
enum : int { ROWS_NONE = 0, ROWS_F16 = 1, ROWS_BF16 = 2, ROWS_GEMM = 3, ROWS_GEMM_Z = 4 };
// Inputs k0 .. k0 + 3 (k0 = 4 * thread + const) of a row into xs (hi) and xs + lo_off (lo, unless lo_off is 0). In either order inputs
// i and i + 4 of a word of 8 are neighbours, so two threads exchange halves and each stores 8 bytes. Returns the sum of what was
// stored (for the zero-point form). All lanes of the warp call it.
template <int MODE>
__device__ __forceinline__ float store_split4(const float (&f)[4], int k0, uint16_t* __restrict__ xs, int lo_off) {
    constexpr bool F16 = MODE == ROWS_F16 || MODE == ROWS_GEMM;
    const bool odd = k0 & 4;
    const int at = MODE >= ROWS_GEMM ? kslot<MODE == ROWS_GEMM_Z>(k0 & ~7) + (odd ? 16 : 0) : split_pos(k0 & ~7) + (odd ? 4 : 0);
    uint16_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) split_hi_lo<F16>(f[i], h[i], l[i]);
    auto put = [&](uint16_t* d, const uint16_t (&w)[4]) {
        const uint32_t p = w[0] | (uint32_t)w[1] << 16, q = w[2] | (uint32_t)w[3] << 16;
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? p : q, 1);
        const uint32_t a = odd ? got : p, b = odd ? q : got;   // inputs (i, i + 1) and (i + 4, i + 5), i = 0 or 2
        *reinterpret_cast<uint2*>(d) = make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
    };
    put(xs + at, h);
    if (lo_off) put(xs + lo_off + at, l);
    float sum = 0.f;
    if constexpr (MODE == ROWS_GEMM_Z)
#pragma unroll
        for (int i = 0; i < 4; i++) { sum += __uint_as_float((uint32_t)h[i] << 16); if (lo_off) sum += __uint_as_float((uint32_t)l[i] << 16); }
    return sum;
}
__device__ __forceinline__ float4 ld_x4(const float* x) { return __ldg(reinterpret_cast<const float4*>(x)); }
// (two 4-byte loads: bf16 rows of a caller are 4-byte aligned, no more)
__device__ __forceinline__ float4 ld_x4(const __nv_bfloat16* x) {
    const uint2 u = make_uint2(__ldg(reinterpret_cast<const uint32_t*>(x)), __ldg(reinterpret_cast<const uint32_t*>(x) + 1));
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xFFFF0000u));
}

}  // namespace moexb
