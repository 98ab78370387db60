// Shared device helpers for the sm_100a denoise-path kernels.
//
// Arithmetic policy: every fused norm / quantise / activation kernel in this
// library computes with explicitly rounded IEEE-754 fp32 operations
// (__fmul_rn, __fadd_rn, __fmaf_rn, __fdiv_rn, __fsqrt_rn) in a fixed order,
// so that a plain-C restatement of the same sequence reproduces every output
// byte.  No fast-math, no approximate reciprocal / rsqrt / exp in those
// kernels.  (GEMM and attention kernels are floating-point kernels with a
// stated tolerance and may use approximate exp2.)
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define FRT_OK 0
#define FRT_ERR_INVALID (-1)
#define FRT_ERR_UNSUPPORTED (-2)
#define FRT_ERR_TIMEOUT (-3)
#define FRT_CUDA_ERR(e) (-(1000 + (int)(e)))

#define FRT_CHECK_LAUNCH()                                  \
    do {                                                    \
        cudaError_t _e = cudaGetLastError();                \
        if (_e != cudaSuccess) return FRT_CUDA_ERR(_e);     \
    } while (0)

namespace frt {

// ---------------------------------------------------------------- bf16 <-> f32
__device__ __forceinline__ float bf16_bits_to_f32(uint32_t b16) {
    return __uint_as_float(b16 << 16);
}
__device__ __forceinline__ void unpack_bf16x2(uint32_t w, float& lo, float& hi) {
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xffff0000u);
}
// round-to-nearest-even fp32 -> bf16, returned in the low 16 bits
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float f) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f));
}
// both halves in one conversion: two scalar ones and an or go through the slow transcendental pipe (one instruction per
// value there in the LayerNorm kernel's profile)
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// v rounded to bf16, as fp32: the upper half of a packed conversion whose lower half is zero IS the fp32 value
__device__ __forceinline__ float bf16_round(float v) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v), "f"(0.0f));
    return __uint_as_float(r);
}

// two fp32 values in one register pair: one instruction for two correctly rounded products or fmas
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f32x2_parts(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t unpack_bf16x2(uint32_t w) {
    return f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// larger magnitude of each half (a NaN loses), its sign the xor of both
__device__ __forceinline__ uint32_t absmax_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// ---------------------------------------------------------------- fp8 e4m3
// clamp to +-448 (NaN -> -448, as fminf(fmaxf(v, -448), 448) gives) in front of a saturating E4M3 conversion: the
// conversion itself does the upper bound, so one instruction remains
__device__ __forceinline__ float clamp448(float v) { return fmaxf(v, -448.0f); }
__device__ __forceinline__ uint32_t f32x2_to_e4m3x2(float lo, float hi) {
    // low byte = lo, high byte = hi
    return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ uint32_t f32x4_to_e4m3x4(float a, float b, float c, float d) {
    return f32x2_to_e4m3x2(a, b) | (f32x2_to_e4m3x2(c, d) << 16);
}

// ---------------------------------------------------------------- exp
// e^x from correctly rounded fp32 operations only (Cody-Waite reduction by
// ln2 in two pieces, degree-7 Taylor/Horner on |r| <= ln2/2, exact scaling by
// 2^n).  The C oracle carries the identical sequence.
__device__ __forceinline__ float det_expf(float x) {
    x = fminf(fmaxf(x, -87.0f), 88.0f);
    float n = rintf(__fmul_rn(x, 1.4426950408889634f));
    float r = __fmaf_rn(n, -0.693145751953125f, x);            // ln2 high part (exact in 12 bits)
    r = __fmaf_rn(n, -1.4286068203094173e-06f, r);             // ln2 low part
    float p = 1.9841269841269841e-04f;                         // 1/5040
    p = __fmaf_rn(p, r, 1.3888888888888889e-03f);              // 1/720
    p = __fmaf_rn(p, r, 8.3333333333333332e-03f);              // 1/120
    p = __fmaf_rn(p, r, 4.1666666666666664e-02f);              // 1/24
    p = __fmaf_rn(p, r, 1.6666666666666666e-01f);              // 1/6
    p = __fmaf_rn(p, r, 0.5f);
    p = __fmaf_rn(p, r, 1.0f);
    p = __fmaf_rn(p, r, 1.0f);
    float s = __int_as_float(((int)n + 127) << 23);            // 2^n, n in [-126,127]
    return __fmul_rn(p, s);
}

// tanh-approximated GELU written as x * sigmoid(2u), u = 0.79788456*(x + 0.044715 x^3)
//   gelu(g) = g / (1 + exp(-1.5957691216057308 * g * (1 + 0.044715 g^2)))
__device__ __forceinline__ float det_gelu_tanh(float g) {
    float inner = __fmaf_rn(__fmul_rn(0.044715f, g), g, 1.0f);
    float arg = __fmul_rn(__fmul_rn(-1.5957691216057308f, g), inner);
    float e = det_expf(arg);
    return __fdiv_rn(g, __fadd_rn(1.0f, e));
}

// The same of two values, bit for bit, with half the instructions: products, fmas and additions run in pairs, round-to-integer is an
// addition of 1.5 * 2^23 (whose sum's low bits are also the exponent of 2^n), and the quotient is Markstein's (IBM J. Res. Dev. 34,
// 1990): reciprocal approximation, one Newton step, quotient, exact remainder, one correction -- correctly rounded as long as
// nothing leaves the normal range, so gates outside 2^-60 <= |g| < 9 (zeros, tiny ones, infinities, NaN, large ones) take the scalar
// form.  Inputs are bf16 values: every finite one is checked against it.
__device__ __forceinline__ uint64_t det_gelu_tanh2(uint64_t g) {
    auto both = [](float v) { return f32x2(v, v); };
    float g0, g1, x0, x1, t0, t1, d0, d1;
    f32x2_parts(g, g0, g1);
    if (!(fabsf(g0) >= 8.673617379884035e-19f && fabsf(g0) < 9.0f && fabsf(g1) >= 8.673617379884035e-19f && fabsf(g1) < 9.0f))
        return f32x2(det_gelu_tanh(g0), det_gelu_tanh(g1));
    const uint64_t one = both(1.0f);
    const uint64_t inner = fma_f32x2(mul_f32x2(both(0.044715f), g), g, one);
    f32x2_parts(mul_f32x2(mul_f32x2(both(-1.5957691216057308f), g), inner), x0, x1);
    const uint64_t x = f32x2(fminf(fmaxf(x0, -87.0f), 88.0f), fminf(fmaxf(x1, -87.0f), 88.0f));
    const uint64_t t = add_f32x2(mul_f32x2(x, both(1.4426950408889634f)), both(12582912.0f));
    const uint64_t n = add_f32x2(t, both(-12582912.0f));
    uint64_t r = fma_f32x2(n, both(-0.693145751953125f), x);
    r = fma_f32x2(n, both(-1.4286068203094173e-06f), r);
    uint64_t p = both(1.9841269841269841e-04f);
    p = fma_f32x2(p, r, both(1.3888888888888889e-03f));
    p = fma_f32x2(p, r, both(8.3333333333333332e-03f));
    p = fma_f32x2(p, r, both(4.1666666666666664e-02f));
    p = fma_f32x2(p, r, both(1.6666666666666666e-01f));
    p = fma_f32x2(p, r, both(0.5f));
    p = fma_f32x2(p, r, one);
    p = fma_f32x2(p, r, one);
    f32x2_parts(t, t0, t1);
    const uint64_t s = f32x2(__uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u),
                             __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u));
    const uint64_t d = add_f32x2(one, mul_f32x2(p, s)), nd = mul_f32x2(d, both(-1.0f));
    f32x2_parts(d, d0, d1);
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(d0));
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(d1));
    uint64_t y = f32x2(d0, d1);
    y = fma_f32x2(y, fma_f32x2(nd, y, one), y);
    const uint64_t q = mul_f32x2(g, y);
    return fma_f32x2(fma_f32x2(nd, q, g), y, q);
}

// SiLU: g * sigmoid(g) = g / (1 + exp(-g))  (silu_mul_split_fp8_kernel, csrc/kernels/activation.cu:291-306)
__device__ __forceinline__ float det_silu(float g) {
    return __fdiv_rn(g, __fadd_rn(1.0f, det_expf(-g)));
}
// GELU(tanh) with the hardware tanh (tanh.approx.f32, relative error 2^-11): 0.5 g (1 + tanh(0.79788456 g (1 + 0.044715 g^2))).
// Six instructions instead of about thirty; not reproducible bit for bit on a CPU, hence an option beside det_gelu_tanh.
// (The reference's kernel is itself built on the fast __expf: csrc/kernels/activation.cu:249-266.)
__device__ __forceinline__ float fast_gelu_tanh(float g) {
    const float u = __fmul_rn(__fmul_rn(0.7978845608028654f, g), __fmaf_rn(__fmul_rn(0.044715f, g), g, 1.0f));
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    return __fmul_rn(__fmul_rn(0.5f, g), __fadd_rn(1.0f, t));
}

// gate activation of the gated FFN epilogues: 0 = GELU(tanh) (GeGLU), 1 = SiLU (SwiGLU)
template <int ACT>
__device__ __forceinline__ uint64_t det_gate_act2(uint64_t g) {
    if (ACT == 0) return det_gelu_tanh2(g);
    float g0, g1;
    f32x2_parts(g, g0, g1);
    return f32x2(det_silu(g0), det_silu(g1));
}

// ---------------------------------------------------------------- reductions
// xor-butterfly: every lane ends with the same value; tree order is fixed.
__device__ __forceinline__ float warp_sum_butterfly(float v) {
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return v;
}
__device__ __forceinline__ float warp_max_butterfly(float v) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return v;
}

// One warp per row: the same sum as "butterfly per 256-column warp slice, then the slices in order" (the tree of the
// one-CTA-per-row kernels and of the C oracle), for a row whose slices all live in ONE warp -- part[w] is this lane's
// partial of slice w.  The butterflies of all slices run together: at every exchange distance a lane keeps half of the
// slices it still holds and hands its partner the other half, so NS slices cost about NS + 5 shuffles instead of 5 * NS
// (every addition keeps its two operands, and an IEEE addition commutes: same bits).  Slices from `n` on do not enter the
// total.
template <int NS>
__device__ __forceinline__ float warp_row_total(const float (&part)[NS], int n) {
    constexpr int P = NS <= 1 ? 1 : NS <= 2 ? 2 : NS <= 4 ? 4 : NS <= 8 ? 8 : NS <= 16 ? 16 : 32;
    static_assert(NS <= 32, "at most 32 slices of 256 columns");
    const int lane = threadIdx.x & 31;
    float v[P];
#pragma unroll
    for (int i = 0; i < P; ++i) v[i] = i < NS ? part[i] : 0.0f;
    int d = 16;
#pragma unroll
    for (int h = P / 2; h >= 1; h >>= 1, d >>= 1) {
        const bool up = (lane & d) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float keep = up ? v[i + h] : v[i], give = up ? v[i] : v[i + h];
            v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, d));
        }
    }
#pragma unroll
    for (; d >= 1; d >>= 1) v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], d));
    float tot = __shfl_sync(0xffffffffu, v[0], 0);
#pragma unroll
    for (int w = 1; w < NS; ++w) {
        const float x = __shfl_sync(0xffffffffu, v[0], w * (32 / P));
        if (w < n) tot = __fadd_rn(tot, x);
    }
    return tot;
}

// The same total for a row whose lanes hold 16 neighbouring values per piece of 512 columns, NP pieces in this warp and WPR warps of
// the row (piece i of warp `part` is i * WPR + part): part0 / part1 are the lane's partials of its first and second eight values.
// A lane holds chunks 2 lane and 2 lane + 1 of a piece's 64, so the exchanges at distance 16, 8, 4, 2 of a chunk are 8, 4, 2, 1 of a
// lane, and the last one is between the halves.  WPR > 1: `slices` = 2 * NP * WPR floats of shared memory for this row, and every
// thread of the block has to come here.
template <int NP, int WPR>
__device__ __forceinline__ float piece_row_total(const float (&part0)[NP], const float (&part1)[NP], int n, int part,
                                                 float* slices) {
    constexpr int P = NP <= 1 ? 1 : NP <= 2 ? 2 : NP <= 4 ? 4 : 8;
    static_assert(NP <= 8 && (WPR == 1 || WPR == 2 || WPR == 4), "pieces per warp, warps per row");
    const int lane = threadIdx.x & 31;
    float v[2 * P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
        v[i] = i < NP ? part0[i < NP ? i : 0] : 0.0f;
        v[P + i] = i < NP ? part1[i < NP ? i : 0] : 0.0f;
    }
    int d = 8;
#pragma unroll
    for (int h = P; h >= 1; h >>= 1, d >>= 1) {
        const bool up = (lane & d) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float keep = up ? v[i + h] : v[i], give = up ? v[i] : v[i + h];
            v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, d));
        }
    }
#pragma unroll
    for (; d >= 1; d >>= 1) v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], d));
    v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], 8));
    // slice 2 (i WPR + part) is in lanes i * (8 / P) .., the one behind it 16 lanes further on
    float tot = 0.0f;
    if (WPR == 1) {
        tot = __shfl_sync(0xffffffffu, v[0], 0);
#pragma unroll
        for (int w = 1; w < 2 * NP; ++w) {
            const float y = __shfl_sync(0xffffffffu, v[0], (w >> 1) * (8 / P) + (w & 1) * 16);
            if (w < n) tot = __fadd_rn(tot, y);
        }
    } else {
        const int i = (lane & 7) / (8 / P);
        if ((lane & 8) == 0 && (lane & 7) % (8 / P) == 0 && i < NP) slices[2 * (i * WPR + part) + (lane >> 4)] = v[0];
        __syncthreads();
        tot = slices[0];
#pragma unroll
        for (int w = 1; w < 2 * NP * WPR; ++w) {
            const float y = slices[w];
            if (w < n) tot = __fadd_rn(tot, y);
        }
    }
    return tot;
}

// Element of every bf16 GEMM epilogue: alpha * acc, or alpha * acc + bias with ONE rounding.  Written out so that every
// kernel that can serve a shape produces the same bits (the compiler is otherwise free to fuse or not, site by site).
__device__ __forceinline__ float scale_bias(float acc, float alpha, float bias, bool has_bias) {
    return has_bias ? __fmaf_rn(acc, alpha, bias) : __fmul_rn(acc, alpha);
}

// Device addresses of the three status words (each lives in the translation unit of its kernels); nullptr on error.
int* gemm_status_device_ptr();
int* attention_status_device_ptr();
int* expert_loop_status_device_ptr();

// ---------------------------------------------------------------- 16-byte I/O
__device__ __forceinline__ uint4 ld_global_v4(const void* p) {
    return *reinterpret_cast<const uint4*>(p);
}
// streaming (read-once) 16-byte load that does not allocate in L1.  A coherent load: the non-coherent form (.nc) promises that
// nobody writes the data while the kernel lives, and a kernel launched programmatically lives before its producer has ended
// (some callers also write the row back in the same kernel).
__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}
// 32 bytes: one instruction where the pointer is 32-byte aligned (`wide`), else two of 16, the second one only if it is there
__device__ __forceinline__ void ld_stream_32(const void* p, bool wide, bool second, uint32_t* r) {
    if (wide) {
        asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "l"(p) : "memory");
    } else {
        const uint4 a = ld_stream_v4(p);
        uint4 b = make_uint4(0, 0, 0, 0);
        if (second) b = ld_stream_v4(static_cast<const uint8_t*>(p) + 16);
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    }
}
__device__ __forceinline__ void st_global_32(void* p, bool wide, bool second, const uint32_t* r) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                     "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
    } else {
        *reinterpret_cast<uint4*>(p) = make_uint4(r[0], r[1], r[2], r[3]);
        if (second) *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p) + 16) = make_uint4(r[4], r[5], r[6], r[7]);
    }
}
__device__ __forceinline__ float4 ld_global_f4(const float* p) {
    return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ void st_global_v4(void* p, uint4 v) {
    *reinterpret_cast<uint4*>(p) = v;
}
__device__ __forceinline__ void st_global_v2(void* p, uint2 v) {
    *reinterpret_cast<uint2*>(p) = v;
}

// Programmatic dependent launch: wait for the producer grid's memory, and let the dependent grid start its prologue early.
// Every kernel that waits before its first global access is launched with the programmatic attribute, whether or not the
// caller passed the PDL flag: its CTAs are then set up (barriers, tensor memory, descriptors) while the kernel in front
// drains, about 1 us per launch.  Behind a kernel that never calls launch_dependents the attribute changes nothing.  The
// caller's flag says more: weights, styles and scales do not come from the kernel in front and may be read before the wait
// (`early`).
// Inputs are no `const __restrict__` parameters and are not read with non-coherent loads (.nc, __ldg): loads from such are
// invariant to the compiler, which may then issue them above the wait, and need not see what the kernel in front wrote while
// this one was already resident.
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------- host: per-device launch set-up
// Function attributes (dynamic shared memory size, non-portable cluster size) and the SM count belong to a device,
// not to the process: a launcher sets them once per device ordinal.
struct PerDeviceOnce {
    bool done[64] = {};
    bool need(int& dev) {
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { dev = -1; return true; }
        return !done[dev];
    }
    void set(int dev) { if (dev >= 0 && dev < 64) done[dev] = true; }
};
inline int device_sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return sms[dev] > 0 ? sms[dev] : 148;
}

}  // namespace frt
