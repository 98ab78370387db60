// Small helpers of the denoise path that are not bandwidth- or tensor-bound:
// the 32 <-> 1024 action projections (bf16, K or N = 32), device copies, device
// queries.
//
// Replaces, for sm_100a, the reference entry points
//   GemmRunner::bf16_nn          csrc/bindings.cpp:662-667 (cuBLASLt) for the action in/out projections
//   gpu_copy                     csrc/bindings.cpp:2533-2537
//   get_sm_version               csrc/bindings.cpp:2447-2453
#include "common.cuh"

namespace frt {

// D(M,N) bf16 = A(M,K) . B(K,N) (+ bias(N)) (+ D when accumulate), bf16 operands, fp32 accumulate.
// Block: 32 output columns x 16 K-slices, 2 output rows.  The projections this
// serves move < 100 KB; the shape of the grid only has to cover the machine.
constexpr int SG_COLS = 32, SG_KS = 16, SG_ROWS = 2, SG_KCHUNK = 1024;

// Element of A, rounded to bf16.  Volatile: a plain load of a const operand may be moved above the wait for the kernel that
// writes it.
template <bool A_F32>
__device__ __forceinline__ float load_a(const void* A, size_t i) {
    if (A_F32) return bf16_round(reinterpret_cast<const volatile float*>(A)[i]);
    return bf16_bits_to_f32(reinterpret_cast<const volatile uint16_t*>(A)[i]);
}

// The sums are formed as 16 interleaved K-slices (k mod 16), added in slice order.  Latency bounds these products, so a
// chunk's weights of a thread are all in flight together, before the wait for the kernel in front when they may be (`early`).
template <bool A_F32, bool D_F32>
__global__ void __launch_bounds__(SG_COLS * SG_KS)
small_gemm_bf16_kernel(const void* Av, const __nv_bfloat16* B,
                       void* __restrict__ Dv, const __nv_bfloat16* bias, int M, int N, int K,
                       int accumulate, int early) {
    __nv_bfloat16* D = reinterpret_cast<__nv_bfloat16*>(Dv);
    float* Df = reinterpret_cast<float*>(Dv);
    __shared__ float a_s[SG_ROWS][SG_KCHUNK];
    __shared__ float part[SG_KS][SG_ROWS][SG_COLS];
    constexpr int PER = SG_KCHUNK / SG_KS;
    const int tx = threadIdx.x % SG_COLS;
    const int ks = threadIdx.x / SG_COLS;
    const int n = blockIdx.x * SG_COLS + tx;
    const int m0 = blockIdx.y * SG_ROWS;
    pdl_launch_dependents();     // the dependent kernel still waits for this grid to complete
    if (!early) pdl_wait();
    float acc[SG_ROWS] = {};
    for (int k0 = 0; k0 < K; k0 += SG_KCHUNK) {
        const int kc = K - k0 < SG_KCHUNK ? K - k0 : SG_KCHUNK;
        __nv_bfloat16 b[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int k = ks + i * SG_KS;
            b[i] = k < kc && n < N ? B[(size_t)(k0 + k) * N + n] : __float2bfloat16_rn(0.0f);
        }
        if (k0 == 0) pdl_wait();
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SG_ROWS; ++r) {
#pragma unroll
            for (int i = 0; i < SG_KCHUNK / (SG_COLS * SG_KS); ++i) {
                const int k = threadIdx.x + i * SG_COLS * SG_KS;
                const size_t ai = (size_t)(m0 + r) * K + k0 + k;
                // an fp32 operand is rounded to bf16 first: the projection multiplies bf16 by bf16
                if (k < kc) a_s[r][k] = m0 + r < M ? (load_a<A_F32>(Av, ai)) : 0.0f;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int k = ks + i * SG_KS;
            if (k < kc) {
#pragma unroll
                for (int r = 0; r < SG_ROWS; ++r) acc[r] = fmaf(a_s[r][k], __bfloat162float(b[i]), acc[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < SG_ROWS; ++r) part[ks][r][tx] = acc[r];
    __syncthreads();
    if (ks < SG_ROWS && n < N && m0 + ks < M) {
        const int r = ks;
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < SG_KS; ++q) s += part[q][r][tx];
        if (bias) s += __bfloat162float(bias[n]);
        const size_t o = (size_t)(m0 + r) * N + n;
        if (D_F32) {
            if (accumulate) s += Df[o];
            Df[o] = s;
        } else {
            if (accumulate) s += __bfloat162float(D[o]);
            D[o] = __float2bfloat16_rn(s);
        }
    }
}

// K = 32 (the action in-projection): a thread forms two columns of four rows, its 32 weight pairs in registers, in the slice
// order of the kernel above -- the same bits with one load round trip and no exchange between threads (200 x 1024: 18 us
// as 3200 CTAs of 512 threads before).  N even, B and D 4-byte aligned.
constexpr int SK_K = 32, SK_ROWS = 4, SK_THREADS = 128;
template <bool A_F32, bool D_F32>
__global__ void __launch_bounds__(SK_THREADS)
short_k_gemm_bf16_kernel(const void* Av, const __nv_bfloat16* B, void* __restrict__ Dv,
                         const __nv_bfloat16* bias, int M, int N, int accumulate, int early) {
    __shared__ float a_s[SK_ROWS][SK_K];
    const int n = (blockIdx.x * SK_THREADS + threadIdx.x) * 2;
    const int m0 = blockIdx.y * SK_ROWS;
    const bool live = n < N;
    pdl_launch_dependents();
    if (!early) pdl_wait();
    uint32_t w[SK_K];
#pragma unroll
    for (int k = 0; k < SK_K; ++k) w[k] = live ? *reinterpret_cast<const uint32_t*>(B + (size_t)k * N + n) : 0u;
    pdl_wait();
    {
        const int r = threadIdx.x / SK_K, k = threadIdx.x % SK_K;
        const size_t ai = (size_t)(m0 + r) * SK_K + k;
        a_s[r][k] = m0 + r < M ? (load_a<A_F32>(Av, ai)) : 0.0f;
    }
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int r = 0; r < SK_ROWS; ++r) {
        if (m0 + r >= M) break;
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            float w00, w01, w10, w11;
            unpack_bf16x2(w[q], w00, w01);
            unpack_bf16x2(w[q + 16], w10, w11);
            s0 += fmaf(a_s[r][q + 16], w10, fmaf(a_s[r][q], w00, 0.0f));
            s1 += fmaf(a_s[r][q + 16], w11, fmaf(a_s[r][q], w01, 0.0f));
        }
        if (bias) {
            s0 += __bfloat162float(bias[n]);
            s1 += __bfloat162float(bias[n + 1]);
        }
        const size_t o = (size_t)(m0 + r) * N + n;
        if (D_F32) {
            float* d = reinterpret_cast<float*>(Dv) + o;
            d[0] = accumulate ? s0 + d[0] : s0;
            d[1] = accumulate ? s1 + d[1] : s1;
        } else {
            uint32_t* d = reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(Dv) + o);
            if (accumulate) {
                float d0, d1;
                unpack_bf16x2(*d, d0, d1);
                s0 += d0;
                s1 += d1;
            }
            *d = pack_bf16x2(s0, s1);
        }
    }
}

// ------------------------------------------------------------------ boundary between two Euler steps, one launch
// Per token one CTA of dim / 2 threads; the norms run on its first dim / 8 (8 features each -- the layout of norm_row_kernel):
//   [has_prev]  xn = bf16(adaRMS(x; style_prev))                      final norm of the step that ends
//               noise += xn . W_out + b_out                            action out-projection (pre-scaled by dt) + Euler
//   [has_next]  x = bf16(bf16(noise) . W_in + b_in)                    action in-projection of the step that begins
//               act8 = e4m3(adaRMS(x; style_next) / *scale)            first norm of layer 0
// Every sum is formed in the order of the kernels this replaces (norm_row_kernel: 8-element fma chain, xor butterfly,
// warp totals in order; small_gemm_bf16_kernel: 16 interleaved K-slices, partials added in slice order, then bias, then
// the old value), so the results are theirs bit for bit.  ACTION = 32 columns of the action space.
constexpr int SB_ACTION = 32;

// Latency bounds it (50 CTAs, a chain of two norms and two small products), so the serial stretches are short: one K-slice of
// the out-projection and two columns of the in-projection per thread.  (With dim / 8 threads, four slices and eight columns
// each: 15.3 us per launch in the loop at 50 x 1024, now 6.5.)

// 1 / rms of the row whose 8-feature sums of squares the first dim / 8 threads hold; every thread reaches both barriers
__device__ __forceinline__ float sb_block_rms(float ssq, float* warp_tot, int dim, float eps) {
    const int nwarps = dim >> 8;
    const int warp = threadIdx.x >> 5;
    if (warp < nwarps) ssq = warp_sum_butterfly(ssq);
    __syncthreads();                                    // warp_tot may still be read from the previous use
    if (warp < nwarps && (threadIdx.x & 31) == 0) warp_tot[warp] = ssq;
    __syncthreads();
    float tot = warp_tot[0];
    for (int w = 1; w < nwarps; ++w) tot = __fadd_rn(tot, warp_tot[w]);
    const float var = __fadd_rn(__fdiv_rn(tot, (float)dim), eps);
    return __fdiv_rn(1.0f, __fsqrt_rn(var));
}

__global__ void __launch_bounds__(1024)
step_boundary_kernel(__nv_bfloat16* __restrict__ x, float* __restrict__ noise, const __nv_bfloat16* style_prev,
                     const __nv_bfloat16* w_out, const __nv_bfloat16* b_out, const __nv_bfloat16* w_in,
                     const __nv_bfloat16* b_in, const __nv_bfloat16* style_next, uint8_t* __restrict__ act8,
                     const float* d_scale, int dim, float eps) {
    extern __shared__ float sb_smem[];
    float* a_s = sb_smem;                               // [dim] normalised row, then the new row (bf16 values)
    float* part = a_s + dim;                            // [16][32] K-slice partials of the out-projection
    float* nz = part + 16 * SB_ACTION;                  // [32] action row, rounded to bf16
    float* warp_tot = nz + SB_ACTION;                   // [32]
    __nv_bfloat16* w_s = reinterpret_cast<__nv_bfloat16*>(warp_tot + 32);   // [dim][32] out-projection weights
    const int t = blockIdx.x, tid = threadIdx.x, col = tid * 8, col2 = tid * 2;
    const bool norm_thread = col < dim;
    const size_t roff = (size_t)t * dim + col;
    pdl_launch_dependents();
    if (style_prev) {
        // the out-projection weights do not depend on the kernel in front: all 16-byte loads in flight, into shared memory
        const uint4* src = reinterpret_cast<const uint4*>(w_out);
        uint4* dst = reinterpret_cast<uint4*>(w_s);
#pragma unroll 8
        for (int i = tid; i < dim * SB_ACTION / 8; i += blockDim.x) dst[i] = src[i];
    }
    // so do this thread's two columns of the in-projection weights (32 rows), held in registers across the first half
    uint32_t wrow[SB_ACTION];
    if (style_next) {
#pragma unroll
        for (int k = 0; k < SB_ACTION; ++k) wrow[k] = *reinterpret_cast<const uint32_t*>(w_in + (size_t)k * dim + col2);
    }
    pdl_wait();
    uint4 nsc = make_uint4(0, 0, 0, 0), nsh = nsc;
    if (style_next && norm_thread) {
        nsc = ld_global_v4(style_next + col);
        nsh = ld_global_v4(style_next + dim + col);
    }
    if (style_prev) {
        float r[8], ssq = 0.0f;
        uint4 sc = make_uint4(0, 0, 0, 0), sh = sc;
        if (norm_thread) {
            const uint4 rv = ld_global_v4(x + roff);
            sc = ld_global_v4(style_prev + col);
            sh = ld_global_v4(style_prev + dim + col);
            const uint32_t* rw = &rv.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                unpack_bf16x2(rw[i], r[2 * i], r[2 * i + 1]);
                ssq = __fmaf_rn(r[2 * i], r[2 * i], ssq);
                ssq = __fmaf_rn(r[2 * i + 1], r[2 * i + 1], ssq);
            }
        }
        const float old = tid < SB_ACTION ? noise[(size_t)t * SB_ACTION + tid] : 0.0f;
        const float rms = sb_block_rms(ssq, warp_tot, dim, eps);
        if (norm_thread) {
            const uint32_t* scw = &sc.x;
            const uint32_t* shw = &sh.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float s0, s1, h0, h1;
                unpack_bf16x2(scw[i], s0, s1);
                unpack_bf16x2(shw[i], h0, h1);
                const float n0 = __fmaf_rn(__fmul_rn(__fmul_rn(r[2 * i], rms), 1.0f), __fadd_rn(1.0f, s0), h0);
                const float n1 = __fmaf_rn(__fmul_rn(__fmul_rn(r[2 * i + 1], rms), 1.0f), __fadd_rn(1.0f, s1), h1);
                a_s[col + 2 * i] = bf16_round(n0);
                a_s[col + 2 * i + 1] = bf16_round(n1);
            }
        }
        __syncthreads();
        // out-projection: column n, K-slices ks = k mod 16; thread (n, g) forms the slices g, g + groups, ...
        const int n = tid % SB_ACTION, g = tid / SB_ACTION, groups = blockDim.x / SB_ACTION;
        for (int ks = g; ks < 16; ks += groups) {
            float acc = 0.0f;
#pragma unroll 16
            for (int k = ks; k < dim; k += 16) acc = fmaf(a_s[k], __bfloat162float(w_s[k * SB_ACTION + n]), acc);
            part[ks * SB_ACTION + n] = acc;
        }
        __syncthreads();
        if (tid < SB_ACTION) {
            float s = 0.0f;
#pragma unroll
            for (int q = 0; q < 16; ++q) s += part[q * SB_ACTION + tid];
            if (b_out) s += __bfloat162float(b_out[tid]);
            s += old;
            noise[(size_t)t * SB_ACTION + tid] = s;
            nz[tid] = bf16_round(s);
        }
    } else if (tid < SB_ACTION) {
        nz[tid] = bf16_round(noise[(size_t)t * SB_ACTION + tid]);
    }
    if (!style_next) return;
    __syncthreads();
    // in-projection: a = bf16(noise); 16 slices of two terms each, partials added in slice order, then the bias
    {
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const float a0 = nz[q], a1 = nz[q + 16];
            float w00, w01, w10, w11;
            unpack_bf16x2(wrow[q], w00, w01);
            unpack_bf16x2(wrow[q + 16], w10, w11);
            s0 += fmaf(a1, w10, fmaf(a0, w00, 0.0f));
            s1 += fmaf(a1, w11, fmaf(a0, w01, 0.0f));
        }
        if (b_in) {
            float b0, b1;
            unpack_bf16x2(*reinterpret_cast<const uint32_t*>(b_in + col2), b0, b1);
            s0 += b0;
            s1 += b1;
        }
        a_s[col2] = bf16_round(s0);
        a_s[col2 + 1] = bf16_round(s1);
        *reinterpret_cast<uint32_t*>(x + (size_t)t * dim + col2) = pack_bf16x2(s0, s1);
    }
    __syncthreads();
    float xb[8], ssq = 0.0f;
    if (norm_thread) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            xb[i] = a_s[col + i];
            ssq = __fmaf_rn(xb[i], xb[i], ssq);
        }
    }
    const float rms = sb_block_rms(ssq, warp_tot, dim, eps);
    if (!norm_thread) return;
    const float inv_scale = __fdiv_rn(1.0f, *d_scale);
    const uint32_t* scw = &nsc.x;
    const uint32_t* shw = &nsh.x;
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float s0, s1, h0, h1;
        unpack_bf16x2(scw[i], s0, s1);
        unpack_bf16x2(shw[i], h0, h1);
        v[2 * i] = __fmaf_rn(__fmul_rn(__fmul_rn(xb[2 * i], rms), 1.0f), __fadd_rn(1.0f, s0), h0);
        v[2 * i + 1] = __fmaf_rn(__fmul_rn(__fmul_rn(xb[2 * i + 1], rms), 1.0f), __fadd_rn(1.0f, s1), h1);
    }
    uint2 o;
    o.x = f32x4_to_e4m3x4(clamp448(__fmul_rn(v[0], inv_scale)), clamp448(__fmul_rn(v[1], inv_scale)),
                          clamp448(__fmul_rn(v[2], inv_scale)), clamp448(__fmul_rn(v[3], inv_scale)));
    o.y = f32x4_to_e4m3x4(clamp448(__fmul_rn(v[4], inv_scale)), clamp448(__fmul_rn(v[5], inv_scale)),
                          clamp448(__fmul_rn(v[6], inv_scale)), clamp448(__fmul_rn(v[7], inv_scale)));
    st_global_v2(act8 + roff, o);
}

}  // namespace frt

using namespace frt;

extern "C" {

// io: bit0 = A is fp32 (rounded to bf16 on load), bit1 = D is fp32
int frt_b200_gemm_bf16_nn_small(const void* A, const void* B, void* D, const void* bias, int M, int N, int K,
                                int accumulate, int io, int flags, void* stream) {
    if (!A || !B || !D || M < 0 || N <= 0 || K <= 0) return FRT_ERR_INVALID;
    if (M == 0) return FRT_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const __nv_bfloat16* Bp = (const __nv_bfloat16*)B;
    const __nv_bfloat16* bp = (const __nv_bfloat16*)bias;
    const int early = flags & 1;                                  // B is weights: not written by the kernel in front
    const int blocks_m = (M + SK_ROWS - 1) / SK_ROWS;
    cudaError_t e;
    if (K == SK_K && (N & 1) == 0 && blocks_m <= 65535 && (reinterpret_cast<uintptr_t>(B) & 3) == 0 &&
        (reinterpret_cast<uintptr_t>(D) & 3) == 0) {
        cfg.gridDim = dim3((N / 2 + SK_THREADS - 1) / SK_THREADS, blocks_m);
        cfg.blockDim = dim3(SK_THREADS);
        switch (io & 3) {
            case 0: e = cudaLaunchKernelEx(&cfg, short_k_gemm_bf16_kernel<false, false>, A, Bp, D, bp, M, N, accumulate, early); break;
            case 1: e = cudaLaunchKernelEx(&cfg, short_k_gemm_bf16_kernel<true, false>, A, Bp, D, bp, M, N, accumulate, early); break;
            case 2: e = cudaLaunchKernelEx(&cfg, short_k_gemm_bf16_kernel<false, true>, A, Bp, D, bp, M, N, accumulate, early); break;
            default: e = cudaLaunchKernelEx(&cfg, short_k_gemm_bf16_kernel<true, true>, A, Bp, D, bp, M, N, accumulate, early); break;
        }
        return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
    }
    cfg.gridDim = dim3((N + SG_COLS - 1) / SG_COLS, (M + SG_ROWS - 1) / SG_ROWS);
    cfg.blockDim = dim3(SG_COLS * SG_KS);
    switch (io & 3) {
        case 0: e = cudaLaunchKernelEx(&cfg, small_gemm_bf16_kernel<false, false>, A, Bp, D, bp, M, N, K, accumulate, early); break;
        case 1: e = cudaLaunchKernelEx(&cfg, small_gemm_bf16_kernel<true, false>, A, Bp, D, bp, M, N, K, accumulate, early); break;
        case 2: e = cudaLaunchKernelEx(&cfg, small_gemm_bf16_kernel<false, true>, A, Bp, D, bp, M, N, K, accumulate, early); break;
        default: e = cudaLaunchKernelEx(&cfg, small_gemm_bf16_kernel<true, true>, A, Bp, D, bp, M, N, K, accumulate, early); break;
    }
    return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
}

// The launches between two Euler steps of the action-expert loop as one (per token: final adaRMS of the step that ends,
// action out-projection accumulated into the fp32 noise, action in-projection of the step that begins, first adaRMS ->
// FP8 of layer 0): Pi05Pipeline.transformer_decoder, flash_rt/models/pi05/pipeline_rtx.py:1451-1504 (C8 of one step and
// C0 / C1 of the next).  style_prev NULL: only the second half (first step); style_next NULL: only the first half (last
// step).  Bit for bit what frt_b200_norm_bf16 -> frt_b200_gemm_bf16_nn_small (accumulate, fp32 D) ->
// frt_b200_gemm_bf16_nn_small (fp32 A) -> frt_b200_norm_fp8 give.  action_dim == 32, dim % 256 == 0, dim <= 2048.
int frt_b200_step_boundary(void* x, float* noise, const void* style_prev, const void* w_out, const void* b_out,
                           const void* w_in, const void* b_in, const void* style_next, void* act8,
                           const float* d_act_scale, int rows, int dim, int action_dim, float eps, int flags,
                           void* stream) {
    if (!x || !noise || rows < 0 || (!style_prev && !style_next)) return FRT_ERR_INVALID;
    if (style_prev && !w_out) return FRT_ERR_INVALID;
    if (style_next && (!w_in || !act8 || !d_act_scale)) return FRT_ERR_INVALID;
    if (action_dim != SB_ACTION || dim <= 0 || (dim % 256) || dim > 2048) return FRT_ERR_UNSUPPORTED;
    const void* ptrs[] = {x, style_prev, w_in, b_in, style_next};
    for (const void* q : ptrs)
        if (reinterpret_cast<uintptr_t>(q) & 15) return FRT_ERR_INVALID;
    if (reinterpret_cast<uintptr_t>(w_out) & 15) return FRT_ERR_INVALID;
    if (reinterpret_cast<uintptr_t>(act8) & 7) return FRT_ERR_INVALID;
    if (rows == 0) return FRT_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows);
    cfg.blockDim = dim3(dim / 2);
    const size_t smem = (size_t)(dim + 16 * SB_ACTION + 2 * SB_ACTION) * sizeof(float) + (size_t)dim * SB_ACTION * 2;
    static PerDeviceOnce attr_once;
    int attr_dev = 0;
    if (attr_once.need(attr_dev)) {
        cudaError_t ea = cudaFuncSetAttribute(step_boundary_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)((2048 + 16 * SB_ACTION + 2 * SB_ACTION) * sizeof(float) + 2048 * SB_ACTION * 2));
        if (ea != cudaSuccess) return FRT_CUDA_ERR(ea);
        attr_once.set(attr_dev);
    }
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (flags & 1) ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, step_boundary_kernel, (__nv_bfloat16*)x, noise,
                                       (const __nv_bfloat16*)style_prev, (const __nv_bfloat16*)w_out,
                                       (const __nv_bfloat16*)b_out, (const __nv_bfloat16*)w_in,
                                       (const __nv_bfloat16*)b_in, (const __nv_bfloat16*)style_next, (uint8_t*)act8,
                                       d_act_scale, dim, eps);
    return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
}

int frt_b200_copy(void* dst, const void* src, long long nbytes, void* stream) {
    if (!dst || !src || nbytes < 0) return FRT_ERR_INVALID;
    if (nbytes == 0) return FRT_OK;
    cudaError_t e = cudaMemcpyAsync(dst, src, (size_t)nbytes, cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
    return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
}

// compute capability as major*10 + minor (100 on B200), or a negative status
int frt_b200_sm_version(void) {
    int dev = 0, major = 0, minor = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return FRT_CUDA_ERR(e);
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
    return major * 10 + minor;
}

}  // extern "C"
