// NVFP4 device helpers: e2m1 element codes, unsigned-E4M3 block scales and the
// scale-factor layout of the block-scaled GEMM.
//
// Format: values +-{0, .5, 1, 1.5, 2, 3, 4, 6} (4 bits, low nibble = even element),
// one unsigned E4M3 scale per 16 consecutive elements of a row.  Scale bytes live in
// 512-byte atoms of 128 rows x 4 blocks, byte (r % 32) * 16 + ((r % 128) / 32) * 4 + (blk % 4),
// atoms ordered K-fastest: atom = (r / 128) * ceil(K / 64) + blk / 4.  This is the layout
// tcgen05.cp (32x128b.warpx4) moves into tensor memory unchanged, and the one the
// reference writes (csrc/kernels/quantize.cu:476-486; CUTLASS Sm1xxBlockScaledConfig<16>
// at csrc/quantize/quantize_fp4_sfa.cu:191-206).
//
// Two quantiser conventions of the reference are kept, selected by `family`:
//   0: scale = smallest UE4M3 >= amax / 6 (csrc/kernels/nvfp4_convert.cuh:78-105), zero block -> scale 0
//      and inverse 0, element thresholds compared with '<'   (nvfp4_convert.cuh:31-45)
//   1: scale = RN-even E4M3 of max(amax / 6, 1e-12), inverse = 1 / scale, thresholds compared with '<='
//      (csrc/quantize/quantize_fp4_sfa.cu:31-50, 89-108)
// All arithmetic is explicitly rounded IEEE fp32, mirrored by the C oracle.
#pragma once
#include "common.cuh"

namespace frt {
namespace nvfp4 {

__device__ __forceinline__ long long sf_offset(long long row, int blk, int katoms) {
    return ((row >> 7) * katoms + (blk >> 2)) * 512 + (row & 31) * 16 + ((row & 127) >> 5) * 4 + (blk & 3);
}

__device__ __forceinline__ float ue4m3_to_f32(uint32_t c) {
    const int e = (c >> 3) & 0xF, m = c & 7;
    // (1 + m/8) * 2^(e-7) for normals, (m/8) * 2^-6 for e == 0; both exact in fp32
    const float mant = e ? __fadd_rn(1.0f, (float)m * 0.125f) : (float)m * 0.125f;
    return __fmul_rn(mant, __int_as_float((127 + (e ? e - 7 : -6)) << 23));
}

// smallest unsigned-E4M3 value >= v; codes above 240 collapse to 0xFE as in the reference
__device__ __forceinline__ uint32_t ue4m3_ceil(float v) {
    if (!(v > 0.0f)) return 0u;
    if (v > 240.0f) return 0xFEu;
    if (v < 0.015625f) {
        const int m = (int)ceilf(__fmul_rn(v, 512.0f));
        if (m > 7) return 0x08u;
        return (uint32_t)(m < 1 ? 1 : m);
    }
    const uint32_t bits = __float_as_uint(v);
    int ex = (int)((bits >> 23) & 0xFF) - 127 + 7;
    const uint32_t frac = bits & 0x7FFFFFu;
    uint32_t m = frac >> 20;
    if (frac & 0xFFFFFu) ++m;
    if (m >= 8) { m = 0; ++ex; }
    if (ex >= 15) return 0xFEu;
    return ((uint32_t)ex << 3) | m;
}

// RN-even E4M3 (saturating finite) of a non-negative value, and back
__device__ __forceinline__ uint32_t e4m3_rn(float v) {
    return (uint32_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float e4m3_to_f32(uint32_t c) {
    return __half2float(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)c, __NV_E4M3)));
}

// Operand of the hardware e2m1 conversion (round to nearest, ties to the even code), moved off the ties that the two
// conventions decide the other way: family 0 rounds every tie up in magnitude (the hardware rounds 0.25, 1.25, 2.5 and 5
// down), family 1 every tie down (the hardware rounds 0.75, 1.75 and 3.5 up).  NaN (0 * inf of an all-zero block in
// family 1) converts to code 7 as the thresholds of both conventions give.
template <int FAMILY>
__device__ __forceinline__ float e2m1_off_tie(float v) {
    const float a = fabsf(v);
    if (FAMILY == 0) return (a == 0.25f || a == 1.25f || a == 2.5f || a == 5.0f) ? __fmul_rn(v, 1.015625f) : v;
    return (a == 0.75f || a == 1.75f || a == 3.5f) ? __fmul_rn(v, 0.984375f) : v;
}

// a / 6 correctly rounded, for 1e-30 <= a (smaller magnitudes end at the 1e-12 floor of the scale): Markstein's division
// by an invariant divisor -- quotient from the rounded reciprocal, one exact remainder, one correction.
__device__ __forceinline__ float sixth(float a) {
    a = fminf(a, 3.0e38f);                                 // inf: the scale saturates either way
    const float r = 0.16666667163372039794921875f;         // 1 / 6 rounded to nearest
    const float q = __fmul_rn(a, r);
    return __fmaf_rn(__fmaf_rn(-6.0f, q, a), r, q);
}

// Multipliers for bf16 inputs whose hardware conversion decides every tie as the convention does: `lo` for |v| < s (codes
// up to 2), `hi` above.  A bf16 value is either exactly (tie x scale) or at least 1 / 255 (relative) away from it (an 8-bit
// significand against the product of a tie's 3 and a scale's 4 bits), so moving a multiplier by 2^-10 decides ties and
// nothing else.  Family 0 rounds all of them up.  Family 1 rounds a product that EQUALS the tie down, but the rounded
// reciprocal of some scales puts odd ties one ulp above: for significands 1.75 and 1.875 the unmoved multiplier is right
// for all seven ties, for 1.625 for those above 1 (every bf16 value x every scale, checked exhaustively).
template <int FAMILY>
__device__ __forceinline__ float2 inv_off_ties(float inv, float s) {
    if (FAMILY == 0) {
        const float up = __fmul_rn(inv, 1.0009765625f);
        return make_float2(up, up);
    }
    const uint32_t sig = (__float_as_uint(s) >> 20) & 7u;   // leading mantissa bits of the scale
    const float down = __fmul_rn(inv, 0.9990234375f);
    return make_float2(sig >= 6u ? inv : down, sig >= 5u ? inv : down);
}

// scale byte of a block and the scale's fp32 value, from the block's largest magnitude
template <int FAMILY>
__device__ __forceinline__ uint32_t block_scale(float amax, float& s) {
    uint32_t sb;
    if (FAMILY == 0) {
        sb = ue4m3_ceil(__fdiv_rn(amax, 6.0f));
        s = ue4m3_to_f32(sb);
    } else {
        sb = e4m3_rn(fmaxf(sixth(amax), 1e-12f));
        s = e4m3_to_f32(sb);
    }
    return sb;
}
template <int FAMILY>
__device__ __forceinline__ float inverse(float s) {
    return FAMILY == 0 ? (s > 0.0f ? __frcp_rn(s) : 0.0f) : __frcp_rn(s);
}

// Eight values -> four bytes (element 0 in the low nibble of byte 0), four hardware conversions of two values each.
__device__ __forceinline__ uint32_t cvt8(const float* x) {
    uint32_t w;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(w)
        : "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7]));
    return w;
}
// any fp32 values: every product is tested for the ties
template <int FAMILY>
__device__ __forceinline__ uint32_t pack8(const float* v, float inv) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = e2m1_off_tie<FAMILY>(__fmaf_rn(v[i], inv, 0.0f));   // + 0: a zero product is +0
    return cvt8(x);
}
// four values -> two bytes
__device__ __forceinline__ uint16_t cvt4(const float* x) {
    uint16_t w;
    asm("{\n\t.reg .b8 b0, b1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "mov.b16 %0, {b0, b1};\n\t}"
        : "=h"(w)
        : "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]));
    return w;
}
template <int FAMILY>
__device__ __forceinline__ uint16_t pack4(const float* v, float inv) {
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = e2m1_off_tie<FAMILY>(__fmaf_rn(v[i], inv, 0.0f));
    return cvt4(x);
}
// bf16 values of a block with scale s; inv from inv_off_ties
template <int FAMILY>
__device__ __forceinline__ uint32_t pack8_bf16(const float* v, float s, float2 inv) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        x[i] = __fmaf_rn(v[i], FAMILY == 0 ? inv.x : (fabsf(v[i]) < s ? inv.x : inv.y), 0.0f);
    return cvt8(x);
}

template <int FAMILY>
__device__ __forceinline__ uint16_t pack4_bf16(const float* v, float s, float2 inv) {
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        x[i] = __fmaf_rn(v[i], FAMILY == 0 ? inv.x : (fabsf(v[i]) < s ? inv.x : inv.y), 0.0f);
    return cvt4(x);
}

}  // namespace nvfp4
}  // namespace frt
