// Fused (gated-)residual + RMSNorm / adaRMS modulation + FP8 E4M3 (or bf16) output.
//
// Replaces, for sm_100a, the reference kernels
//   rms_norm_fp8                 csrc/kernels/norm.cu:286-343
//   ada_rms_norm_style           csrc/kernels/norm.cu:345-389
//   ada_rms_norm_style_fp8       csrc/kernels/norm.cu:392-442
//   residual_add_rms_norm_fp8    csrc/kernels/norm.cu:445-495
//   residual_add_rms_norm        csrc/kernels/norm.cu:498-539
//   gate_residual_ada_norm_fp8   csrc/kernels/fusion.cu:15-81
//
// Design: one CTA per row, one 16-byte vector (8 bf16) per thread, so a row of
// `dim` elements uses dim/8 threads (rounded up to whole warps).  The row is
// read once and kept in registers: the residual update, its bf16 rounding, the
// sum of squares and the normalisation all happen without a second trip to
// memory.  All loads are 16-byte and coalesced; the FP8 result leaves as one
// 8-byte store per thread, the updated residual as one 16-byte store.
//
// Rounding points kept from the reference: the residual update is computed in
// fp32 and stored as bf16; the sum of squares uses the unrounded fp32 value;
// the normalisation reads the rounded bf16 value; the modulated value is not
// rounded to bf16 before the FP8 conversion; quantisation multiplies by the
// fp32 reciprocal of the scale, clamps to +-448 and converts RN-even.
//
// Reduction tree (fixed, mirrored by the C oracle): per thread a sequential
// fma chain over its 8 elements; xor-butterfly over the 32 lanes; warp totals
// summed in warp order by every thread.
#include "nvfp4.cuh"

namespace frt {

enum { OUT_BF16 = 0, OUT_E4M3 = 1, OUT_NVFP4_A = 2, OUT_NVFP4_B = 3 };

struct NormArgs {
    __nv_bfloat16* residual;       // in/out row-major (rows, dim); or input x when !HAS_X
    const __nv_bfloat16* x;        // sub-layer output to add (HAS_X)
    const __nv_bfloat16* gate_in;  // multiplies x before the add (HAS_GATE)
    long long gate_in_stride;      // elements between gate rows (0 = one shared row)
    const __nv_bfloat16* weight;   // (dim,) or null (= ones)
    const __nv_bfloat16* style;    // rows of [scale | shift | gate], 3*dim each (HAS_STYLE)
    long long style_stride;        // elements between style rows (0 = one shared row)
    void* out;                     // fp8 (rows, dim), bf16 (rows, dim) or packed e2m1 (rows, dim / 2)
    uint8_t* sf_out;               // NVFP4 block scales in the GEMM's scale-factor atoms
    __nv_bfloat16* gate_out;       // copy of the style gate chunk, or null
    const float* d_scale;          // device scalar: quantisation scale (OUT_FP8)
    int rows;
    int dim;
    float eps;
    int early;                     // weight, style and scale may be read before the kernel in front has finished
};

template <bool HAS_X, bool HAS_GATE, bool HAS_STYLE, int OUT>
__global__ void __launch_bounds__(1024)
norm_row_kernel(NormArgs a) {
    constexpr bool OUT_FP8 = OUT == OUT_E4M3;
    constexpr bool OUT_FP4 = OUT == OUT_NVFP4_A || OUT == OUT_NVFP4_B;
    __shared__ float warp_tot[32];
    const int row = blockIdx.x;
    const int tid = threadIdx.x;
    const int col = tid * 8;
    const bool active = col < a.dim;
    const size_t roff = (size_t)row * a.dim + col;

    float r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = 0.0f;
    uint4 wv = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
    uint4 sc = make_uint4(0, 0, 0, 0), sh = sc, gt = sc;

    // The next kernel in the stream may start its own input-independent prologue right away (it still waits for
    // this grid to finish before it touches anything this grid writes).
    pdl_launch_dependents();
    if (!a.early) pdl_wait();
    // Everything that does not depend on the producer kernel is fetched first.
    if (active) {
        if (a.weight) wv = ld_global_v4(a.weight + col);
        if (HAS_STYLE) {
            const __nv_bfloat16* srow = a.style + (size_t)row * a.style_stride;
            sc = ld_global_v4(srow + col);
            sh = ld_global_v4(srow + a.dim + col);
            if (a.gate_out) gt = ld_global_v4(srow + 2 * (size_t)a.dim + col);
        }
    }
    float inv_scale = 1.0f;
    if (OUT_FP8) inv_scale = __fdiv_rn(1.0f, *a.d_scale);

    pdl_wait();

    float ssq = 0.0f;
    uint4 rbits = make_uint4(0, 0, 0, 0);
    if (active) {
        uint4 rv = ld_global_v4(a.residual + roff);
        const uint32_t* rw = &rv.x;
        if (HAS_X) {
            uint4 xv = ld_stream_v4(a.x + roff);
            const uint32_t* xw = &xv.x;
            uint4 gv = make_uint4(0, 0, 0, 0);
            if (HAS_GATE) gv = ld_global_v4(a.gate_in + (size_t)row * a.gate_in_stride + col);
            const uint32_t* gw = &gv.x;
            uint32_t* ow = &rbits.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float r0, r1, x0, x1;
                unpack_bf16x2(rw[i], r0, r1);
                unpack_bf16x2(xw[i], x0, x1);
                if (HAS_GATE) {
                    float g0, g1;
                    unpack_bf16x2(gw[i], g0, g1);
                    r0 = __fmaf_rn(x0, g0, r0);
                    r1 = __fmaf_rn(x1, g1, r1);
                } else {
                    r0 = __fadd_rn(r0, x0);
                    r1 = __fadd_rn(r1, x1);
                }
                ssq = __fmaf_rn(r0, r0, ssq);
                ssq = __fmaf_rn(r1, r1, ssq);
                ow[i] = pack_bf16x2(r0, r1);
                unpack_bf16x2(ow[i], r[2 * i], r[2 * i + 1]);   // rounded value feeds the norm
            }
            st_global_v4(a.residual + roff, rbits);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                unpack_bf16x2(rw[i], r[2 * i], r[2 * i + 1]);
                ssq = __fmaf_rn(r[2 * i], r[2 * i], ssq);
                ssq = __fmaf_rn(r[2 * i + 1], r[2 * i + 1], ssq);
            }
        }
    }
    ssq = warp_sum_butterfly(ssq);
    const int nwarps = blockDim.x >> 5;
    if ((tid & 31) == 0) warp_tot[tid >> 5] = ssq;
    __syncthreads();
    float tot = warp_tot[0];
    for (int w = 1; w < nwarps; ++w) tot = __fadd_rn(tot, warp_tot[w]);
    const float var = __fadd_rn(__fdiv_rn(tot, (float)a.dim), a.eps);
    const float rms = __fdiv_rn(1.0f, __fsqrt_rn(var));

    if (!OUT_FP4 && !active) return;   // the NVFP4 path shuffles between lane pairs: every lane stays

    float v[8];
    const uint32_t* ww = &wv.x;
    const uint32_t* scw = &sc.x;
    const uint32_t* shw = &sh.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float w0, w1;
        unpack_bf16x2(ww[i], w0, w1);
        float n0 = __fmul_rn(__fmul_rn(r[2 * i], rms), w0);
        float n1 = __fmul_rn(__fmul_rn(r[2 * i + 1], rms), w1);
        if (HAS_STYLE) {
            float s0, s1, h0, h1;
            unpack_bf16x2(scw[i], s0, s1);
            unpack_bf16x2(shw[i], h0, h1);
            n0 = __fmaf_rn(n0, __fadd_rn(1.0f, s0), h0);
            n1 = __fmaf_rn(n1, __fadd_rn(1.0f, s1), h1);
        }
        v[2 * i] = n0;
        v[2 * i + 1] = n1;
    }
    if (OUT_FP4) {
        // The modulated value is rounded to bf16 (what the bf16-output kernel stores) and then quantised in
        // blocks of 16 = this thread's 8 values and its lane neighbour's; the even lane writes the scale byte.
        constexpr int FAM = OUT == OUT_NVFP4_A ? 0 : 1;
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            unpack_bf16x2(pack_bf16x2(v[i], v[i + 1]), v[i], v[i + 1]);
            amax = fmaxf(amax, fmaxf(fabsf(v[i]), fabsf(v[i + 1])));
        }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        float s;
        const uint32_t sb = nvfp4::block_scale<FAM>(amax, s);
        const float2 inv = nvfp4::inv_off_ties<FAM>(nvfp4::inverse<FAM>(s), s);
        if (active) {
            *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(a.out) + (roff >> 1)) = nvfp4::pack8_bf16<FAM>(v, s, inv);
            if ((tid & 1) == 0) a.sf_out[nvfp4::sf_offset(row, col >> 4, (a.dim + 63) >> 6)] = (uint8_t)sb;
            if (HAS_STYLE && a.gate_out) st_global_v4(a.gate_out + roff, gt);
        }
        return;
    }
    if (OUT_FP8) {
        uint2 o;
        o.x = f32x4_to_e4m3x4(clamp448(__fmul_rn(v[0], inv_scale)), clamp448(__fmul_rn(v[1], inv_scale)),
                              clamp448(__fmul_rn(v[2], inv_scale)), clamp448(__fmul_rn(v[3], inv_scale)));
        o.y = f32x4_to_e4m3x4(clamp448(__fmul_rn(v[4], inv_scale)), clamp448(__fmul_rn(v[5], inv_scale)),
                              clamp448(__fmul_rn(v[6], inv_scale)), clamp448(__fmul_rn(v[7], inv_scale)));
        st_global_v2(reinterpret_cast<uint8_t*>(a.out) + roff, o);
    } else {
        uint4 o;
        o.x = pack_bf16x2(v[0], v[1]);
        o.y = pack_bf16x2(v[2], v[3]);
        o.z = pack_bf16x2(v[4], v[5]);
        o.w = pack_bf16x2(v[6], v[7]);
        st_global_v4(reinterpret_cast<__nv_bfloat16*>(a.out) + roff, o);
    }
    if (HAS_STYLE && a.gate_out) st_global_v4(a.gate_out + roff, gt);
}

// Many rows: a warp, or WPR of the CTA's four warps, takes a row; it stays in registers, 16 neighbouring values per lane and piece
// of 512 columns, NP pieces per warp.  The one-CTA-per-row kernel above is bound by its latency chain -- one load, one block barrier
// and a serial sum of warp totals per row, a few rows on an SM.  Here every lane has NP loads of 32 bytes in flight and 16-24 rows
// share an SM.  A lane's 16 values are one block of the NVFP4 result, whose scale, reciprocal and conversions are then made once
// (twice with 8 values per lane), products and fmas run two at a time, the largest magnitude on packed bf16: what bounds the
// NVFP4 result is still its instructions, about 95 per 8 values.  Same sums in the same order as the CTA kernel, same bits.
// us, one warp per row with 8 values per lane (above 4096 columns: one CTA per row) -> now: to NVFP4 20480 x 3072 59.8 -> 45.2, 8192
// x 8192 101 -> 50, 2501 x 3072 11.4 -> 8.7; to FP8 20480 x 3072 34.2 -> 32.5 (5.8 TB/s), 8192 x 4096 22.5 -> 19.7, 8192 x 8192 84.8 ->
// 36.7; to bf16 (a lane's 32 bytes as one store; as two, every store touches half of each sector: 4096 x 4096 11.8 instead of 10.6)
// 8192 x 4096 24.3 -> 21.4.
template <int OUT, int NP, int WPR>
__global__ void __launch_bounds__(128)
norm_block_kernel(NormArgs a) {
    constexpr bool OUT_FP8 = OUT == OUT_E4M3;
    constexpr bool OUT_FP4 = OUT == OUT_NVFP4_A || OUT == OUT_NVFP4_B;
    constexpr uint32_t HI = 0xffff0000u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = blockIdx.x * (4 / WPR) + warp / WPR, part = warp % WPR;
    pdl_launch_dependents();
    pdl_wait();
    const float inv_scale = OUT_FP8 ? __fdiv_rn(1.0f, *a.d_scale) : 1.0f;
    const bool live = row < a.rows;
    if (WPR == 1 && !live) return;
    // whole: every lane's piece is 32 bytes at a multiple of 32, its result one aligned store; otherwise by halves of 8 values
    const bool wide = ((reinterpret_cast<uintptr_t>(a.residual) & 31) | (a.dim & 15)) == 0;
    const bool whole = ((reinterpret_cast<uintptr_t>(a.out) & (OUT == OUT_BF16 ? 31 : 15)) | (a.dim & 15)) == 0;
    const int col0 = part * 512 + lane * 16;                // pair i of this lane: columns col0 + i * WPR * 512 ..
    const size_t rbase = (size_t)row * a.dim + col0;
    const int left = live ? a.dim - col0 : 0;
    uint32_t x[NP][8];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[i][j] = 0u;
        if (i * WPR * 512 < left) ld_stream_32(a.residual + rbase + i * WPR * 512, wide, i * WPR * 512 + 8 < left, x[i]);
    }
    // sums of squares, the chains over the 8 values of both halves at once
    float part0[NP], part1[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        uint64_t s = f32x2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t e = f32x2(__uint_as_float(x[i][j] << 16), __uint_as_float(x[i][4 + j] << 16));
            const uint64_t o = f32x2(__uint_as_float(x[i][j] & HI), __uint_as_float(x[i][4 + j] & HI));
            s = fma_f32x2(o, o, fma_f32x2(e, e, s));
        }
        f32x2_parts(s, part0[i], part1[i]);
    }
    __shared__ float slices[WPR == 1 ? 1 : 4 / WPR][WPR == 1 ? 1 : 2 * NP * WPR];
    const float tot = piece_row_total<NP, WPR>(part0, part1, (a.dim + 255) >> 8, part, slices[WPR == 1 ? 0 : warp / WPR]);
    if (!live) return;
    const float var = __fadd_rn(__fdiv_rn(tot, (float)a.dim), a.eps);
    const float rms = __fdiv_rn(1.0f, __fsqrt_rn(var));
    const uint64_t rms2 = f32x2(rms, rms), zero2 = f32x2(0.0f, 0.0f);
    uint8_t* sf = nullptr;                                  // scale byte of this lane's block of pair 0
    const bool sf_words = OUT_FP4 && (a.dim & 63) == 0;
    if (OUT_FP4) sf = a.sf_out + nvfp4::sf_offset(row, (part * 32 + lane) & ~3, (a.dim + 63) >> 6);
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const bool on = i * WPR * 512 < left, on2 = i * WPR * 512 + 8 < left;
        uint32_t wv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) wv[j] = 0x3f803f80u;
        if (on && a.weight) {
            const __nv_bfloat16* wp = a.weight + col0 + i * WPR * 512;
            const uint4 w0 = ld_global_v4(wp), w1 = on2 ? ld_global_v4(wp + 8) : w0;
            wv[0] = w0.x; wv[1] = w0.y; wv[2] = w0.z; wv[3] = w0.w;
            wv[4] = w1.x; wv[5] = w1.y; wv[6] = w1.z; wv[7] = w1.w;
        }
        uint64_t y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = mul_f32x2(mul_f32x2(unpack_bf16x2(x[i][j]), rms2), unpack_bf16x2(wv[j]));
        const size_t roff = rbase + i * WPR * 512;
        if (OUT_FP8) {
            const uint64_t is2 = f32x2(inv_scale, inv_scale);
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float q0, q1, q2, q3;
                f32x2_parts(mul_f32x2(y[2 * j], is2), q0, q1);
                f32x2_parts(mul_f32x2(y[2 * j + 1], is2), q2, q3);
                o[j] = f32x4_to_e4m3x4(clamp448(q0), clamp448(q1), clamp448(q2), clamp448(q3));
            }
            uint8_t* dst = reinterpret_cast<uint8_t*>(a.out) + roff;
            if (whole) {
                if (on) st_global_v4(dst, make_uint4(o[0], o[1], o[2], o[3]));
            } else {
                if (on) st_global_v2(dst, make_uint2(o[0], o[1]));
                if (on2) st_global_v2(dst + 8, make_uint2(o[2], o[3]));
            }
            continue;
        }
        uint32_t b[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float y0, y1;
            f32x2_parts(y[j], y0, y1);
            b[j] = pack_bf16x2(y0, y1);
        }
        if (!OUT_FP4) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + roff;
            if (on) st_global_32(dst, whole, on2, b);
            continue;
        }
        constexpr int FAM = OUT == OUT_NVFP4_A ? 0 : 1;
        const uint32_t m = absmax_bf16x2(absmax_bf16x2(absmax_bf16x2(b[0], b[1]), absmax_bf16x2(b[2], b[3])),
                                         absmax_bf16x2(absmax_bf16x2(b[4], b[5]), absmax_bf16x2(b[6], b[7]))) & 0x7fff7fffu;
        const float amax = fmaxf(0.0f, fmaxf(__uint_as_float(m << 16), __uint_as_float(m & HI)));
        float s;
        uint32_t sb = nvfp4::block_scale<FAM>(amax, s);
        const float2 inv = nvfp4::inv_off_ties<FAM>(nvfp4::inverse<FAM>(s), s);
        uint32_t q[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float e[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float y0, y1;
                f32x2_parts(unpack_bf16x2(b[4 * h + j]), y0, y1);
                const uint64_t i2 = FAM == 0 ? f32x2(inv.x, inv.x)
                                             : f32x2(fabsf(y0) < s ? inv.x : inv.y, fabsf(y1) < s ? inv.x : inv.y);
                f32x2_parts(fma_f32x2(f32x2(y0, y1), i2, zero2), e[2 * j], e[2 * j + 1]);
            }
            q[h] = nvfp4::cvt8(e);
        }
        if (on) st_global_v2(reinterpret_cast<uint8_t*>(a.out) + (roff >> 1), make_uint2(q[0], q[1]));
        // the scale bytes of four neighbouring blocks (lanes) are one aligned word of the scale layout
        if (sf_words) {
            sb |= __shfl_down_sync(0xffffffffu, sb, 1) << 8;
            sb |= __shfl_down_sync(0xffffffffu, sb, 2) << 16;
            if (on && (lane & 3) == 0) *reinterpret_cast<uint32_t*>(sf + i * WPR * 4096) = sb;
        } else if (on) {
            sf[i * WPR * 4096 + (lane & 3)] = (uint8_t)sb;
        }
    }
}

// FP8 and bf16, many short rows: one warp per row with 8 values per lane and slice of 256 columns (NS slices).  What bounds these is
// the loads in flight, and with 16 values per lane a short row's last piece is half empty and its results take twice the registers:
// 20480 x 768 to bf16 10.2 us there and 9.3 here, 4096 x 1024 4.2 and 3.7, 20480 x 1280 to FP8 14.9 and 13.9.  Same sums, same bits.
template <int OUT, int NS>
__global__ void __launch_bounds__(128)
norm_warp_kernel(NormArgs a) {
    static_assert(OUT == OUT_BF16 || OUT == OUT_E4M3, "results of one value per element");
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
    pdl_launch_dependents();
    pdl_wait();
    const float inv_scale = OUT == OUT_E4M3 ? __fdiv_rn(1.0f, *a.d_scale) : 1.0f;
    if (row >= a.rows) return;
    const int n = (a.dim + 255) >> 8;                       // slices of this row, n <= NS
    const size_t rbase = (size_t)row * a.dim + lane * 8;
    const int left = a.dim - lane * 8;                      // slice w of this lane exists while w * 256 < left
    uint4 rv[NS];
    float ssq[NS];
#pragma unroll
    for (int w = 0; w < NS; ++w) {
        rv[w] = make_uint4(0, 0, 0, 0);
        if (w * 256 < left) rv[w] = ld_stream_v4(a.residual + rbase + w * 256);
    }
#pragma unroll
    for (int w = 0; w < NS; ++w) {
        const uint32_t* rw = &rv[w].x;
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float r0, r1;
            unpack_bf16x2(rw[i], r0, r1);
            s = __fmaf_rn(r0, r0, s);
            s = __fmaf_rn(r1, r1, s);
        }
        ssq[w] = s;
    }
    const float tot = warp_row_total<NS>(ssq, n);
    const float var = __fadd_rn(__fdiv_rn(tot, (float)a.dim), a.eps);
    const float rms = __fdiv_rn(1.0f, __fsqrt_rn(var));
#pragma unroll
    for (int w = 0; w < NS; ++w) {
        const bool on = w * 256 < left;
        uint4 wv = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
        if (on && a.weight) wv = ld_global_v4(a.weight + lane * 8 + w * 256);
        const uint32_t* rw = &rv[w].x;
        const uint32_t* ww = &wv.x;
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float r0, r1, w0, w1;
            unpack_bf16x2(rw[i], r0, r1);
            unpack_bf16x2(ww[i], w0, w1);
            v[2 * i] = __fmul_rn(__fmul_rn(r0, rms), w0);
            v[2 * i + 1] = __fmul_rn(__fmul_rn(r1, rms), w1);
        }
        const size_t roff = rbase + w * 256;
        if (OUT == OUT_E4M3) {
            uint2 o;
            o.x = f32x4_to_e4m3x4(clamp448(__fmul_rn(v[0], inv_scale)), clamp448(__fmul_rn(v[1], inv_scale)),
                                  clamp448(__fmul_rn(v[2], inv_scale)), clamp448(__fmul_rn(v[3], inv_scale)));
            o.y = f32x4_to_e4m3x4(clamp448(__fmul_rn(v[4], inv_scale)), clamp448(__fmul_rn(v[5], inv_scale)),
                                  clamp448(__fmul_rn(v[6], inv_scale)), clamp448(__fmul_rn(v[7], inv_scale)));
            if (on) st_global_v2(reinterpret_cast<uint8_t*>(a.out) + roff, o);
        } else {
            uint4 o;
            o.x = pack_bf16x2(v[0], v[1]);
            o.y = pack_bf16x2(v[2], v[3]);
            o.z = pack_bf16x2(v[4], v[5]);
            o.w = pack_bf16x2(v[6], v[7]);
            if (on) st_global_v4(reinterpret_cast<__nv_bfloat16*>(a.out) + roff, o);
        }
    }
}

// CTAs of 128 threads, `per` rows each
static int launch_norm_rows(void (*kern)(NormArgs), const NormArgs& a, int per, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((a.rows + per - 1) / per));
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
}

// The kernel of an RMSNorm without a residual (null: the one-CTA-per-row kernel) and the rows of its CTA.  Timed at 528 .. 8192
// columns, 256 .. 20480 rows and the three kinds of result; all give the same bits.  What decides is how many rows of a form an
// SM holds, so the lines are in rows per SM (us, the form taken first):
//   above 1536 columns the chain of the CTA kernel counts from 3 Mi values on, when its rows no longer fit the chip at once; below,
//   it is the shorter one (512 x 3072 to NVFP4 3.4 against 4.5).  Two warps per row up to 3072 columns, four above, so that a lane
//   holds two to four pieces (20480 x 4096 to NVFP4 with 4 / 2 / 1 warps: 58 / 64 / 73).  But where five pieces leave one of two warps
//   idle in the third: one warp of 16 values at 13 to 16 rows (2304 x 2560 to FP8 5.2, two warps 6.2), the 8-value kernel up to 20,
//   its full wave, and above 40 (20480 x 2560 to FP8 27.9, two warps 32.3).  Its full wave is also 16 to 20 rows of four pieces (2816 x
//   2048 to bf16 4.5, two warps 5.2) and up to 16 of six (2304 x 3072 to bf16 5.8, two warps 6.8).
//   up to 1536 columns: more than 20 rows take a warp each, with 16 values per lane to NVFP4 (its instructions count) and to FP8 where
//   they fill more than half of the last piece (20480 x 1024 11.2, 8 values 11.6), else with 8; more than 15 take two warps each (2560
//   x 1024 to FP8 2.8, one warp 3.0, the CTA kernel 4.1), but not to NVFP4 above 1024 columns (2560 x 1280: the CTA kernel 5.0, two
//   warps 6.1).
// The residual form stays with the CTA kernel at every size (it already streams 5.6 TB/s; two register-held rows per lane were
// slower).
struct NormRows { void (*kern)(NormArgs); int per; };
template <int OUT>
static NormRows pick_norm_rows(const NormArgs& a) {
    constexpr bool FP4 = OUT == OUT_NVFP4_A || OUT == OUT_NVFP4_B;
    constexpr NormRows CTA = {nullptr, 0};
    const long long rows = a.rows;
    const int pieces = (a.dim + 511) / 512;
    const bool values = rows * a.dim >= 3ll << 20;
    if (rows < 512 && !values) return CTA;              // below every line: the smallest calls are spared the question (0.03 us)
    const long long sms = device_sm_count();
    if (a.dim <= 512 || (FP4 && ((reinterpret_cast<uintptr_t>(a.sf_out) & 3) || (reinterpret_cast<uintptr_t>(a.out) & 7))))
        return CTA;
    if (pieces > 3) {
        if (!values) return CTA;
        if (pieces > 12) return {norm_block_kernel<OUT, 4, 4>, 1};
        if (pieces > 8) return {norm_block_kernel<OUT, 3, 4>, 1};
        if (pieces > 6) return {norm_block_kernel<OUT, 2, 4>, 1};
        if constexpr (OUT != OUT_BF16)
            if (pieces == 5 && rows > 12 * sms && rows <= 16 * sms) return {norm_block_kernel<OUT, 5, 1>, 4};
        if constexpr (!FP4) {
            if (pieces == 4 && rows > 16 * sms && rows <= 20 * sms) return {norm_warp_kernel<OUT, 8>, 4};
            if (pieces == 5 && rows > 14 * sms && (rows <= 20 * sms || rows > 40 * sms)) return {norm_warp_kernel<OUT, 10>, 4};
            if (pieces == 6 && rows > 14 * sms && rows <= 16 * sms) return {norm_warp_kernel<OUT, 12>, 4};
        }
        if (pieces == 4) return {norm_block_kernel<OUT, 2, 2>, 2};
        return {norm_block_kernel<OUT, 3, 2>, 2};
    }
    if (rows > 20 * sms) {
        if constexpr (!FP4)
            if (OUT == OUT_BF16 || ((a.dim - 1) & 511) < 256)
                return {pieces == 2 ? norm_warp_kernel<OUT, 4> : norm_warp_kernel<OUT, 6>, 4};
        if constexpr (OUT != OUT_BF16)
            return {pieces == 2 ? norm_block_kernel<OUT, 2, 1> : norm_block_kernel<OUT, 3, 1>, 4};
    }
    if (FP4 ? pieces == 2 && rows > 15 * sms : values || rows > 15 * sms)
        return {pieces == 2 ? norm_block_kernel<OUT, 1, 2> : norm_block_kernel<OUT, 2, 2>, 2};
    return CTA;
}

template <bool HAS_X, bool HAS_GATE, bool HAS_STYLE, int OUT>
static int launch_norm(NormArgs a, cudaStream_t stream, bool pdl) {
    a.early = pdl ? 1 : 0;
    if (a.rows < 0 || a.dim <= 0 || (a.dim & 7) || a.dim > 8192) return FRT_ERR_UNSUPPORTED;
    if (a.rows == 0) return FRT_OK;
    if constexpr (!HAS_X && !HAS_STYLE) {
        const NormRows many = pick_norm_rows<OUT>(a);
        if (many.kern) return launch_norm_rows(many.kern, a, many.per, stream);
    }
    int threads = ((a.dim / 8 + 31) / 32) * 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.rows);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, norm_row_kernel<HAS_X, HAS_GATE, HAS_STYLE, OUT>, a);
    if (e != cudaSuccess) return FRT_CUDA_ERR(e);
    return FRT_OK;
}

}  // namespace frt

using namespace frt;

template <int OUT>
static int dispatch_norm_nvfp4(const NormArgs& a, bool has_x, bool has_gate, bool has_style, cudaStream_t s, bool pdl) {
    if (has_x) {
        if (has_gate) {
            if (has_style) return launch_norm<true, true, true, OUT>(a, s, pdl);
            return launch_norm<true, true, false, OUT>(a, s, pdl);
        }
        if (has_style) return launch_norm<true, false, true, OUT>(a, s, pdl);
        return launch_norm<true, false, false, OUT>(a, s, pdl);
    }
    if (has_style) return launch_norm<false, false, true, OUT>(a, s, pdl);
    return launch_norm<false, false, false, OUT>(a, s, pdl);
}

static inline bool misaligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

extern "C" {

// flags: bit0 = launch with programmatic stream serialization (PDL)
int frt_b200_norm_fp8(void* residual, const void* x, const void* gate_in, long long gate_in_stride,
                      const void* weight, const void* style, long long style_stride, void* out_fp8,
                      void* gate_out, int rows, int dim, float eps, const float* d_scale, int flags,
                      void* stream) {
    if (!residual || !out_fp8 || !d_scale) return FRT_ERR_INVALID;
    if (gate_in && !x) return FRT_ERR_INVALID;
    if (misaligned16(residual) || misaligned16(x) || misaligned16(gate_in) || misaligned16(weight) ||
        misaligned16(style) || misaligned16(gate_out) || (reinterpret_cast<uintptr_t>(out_fp8) & 7))
        return FRT_ERR_INVALID;
    if ((gate_in_stride & 7) || (style_stride & 7)) return FRT_ERR_INVALID;
    NormArgs a;
    a.residual = (__nv_bfloat16*)residual;
    a.x = (const __nv_bfloat16*)x;
    a.gate_in = (const __nv_bfloat16*)gate_in;
    a.gate_in_stride = gate_in_stride;
    a.weight = (const __nv_bfloat16*)weight;
    a.style = (const __nv_bfloat16*)style;
    a.style_stride = style_stride;
    a.out = out_fp8;
    a.sf_out = nullptr;
    a.gate_out = (__nv_bfloat16*)gate_out;
    a.d_scale = d_scale;
    a.rows = rows;
    a.dim = dim;
    a.eps = eps;
    cudaStream_t s = (cudaStream_t)stream;
    bool pdl = flags & 1;
    if (x) {
        if (gate_in) {
            if (style) return launch_norm<true, true, true, OUT_E4M3>(a, s, pdl);
            return launch_norm<true, true, false, OUT_E4M3>(a, s, pdl);
        }
        if (style) return launch_norm<true, false, true, OUT_E4M3>(a, s, pdl);
        return launch_norm<true, false, false, OUT_E4M3>(a, s, pdl);
    }
    if (style) return launch_norm<false, false, true, OUT_E4M3>(a, s, pdl);
    return launch_norm<false, false, false, OUT_E4M3>(a, s, pdl);
}

int frt_b200_norm_bf16(void* residual, const void* x, const void* gate_in, long long gate_in_stride,
                       const void* weight, const void* style, long long style_stride, void* out_bf16,
                       void* gate_out, int rows, int dim, float eps, int flags, void* stream) {
    if (!residual || !out_bf16) return FRT_ERR_INVALID;
    if (gate_in && !x) return FRT_ERR_INVALID;
    if (misaligned16(residual) || misaligned16(x) || misaligned16(gate_in) || misaligned16(weight) ||
        misaligned16(style) || misaligned16(gate_out) || misaligned16(out_bf16))
        return FRT_ERR_INVALID;
    if ((gate_in_stride & 7) || (style_stride & 7)) return FRT_ERR_INVALID;
    NormArgs a;
    a.residual = (__nv_bfloat16*)residual;
    a.x = (const __nv_bfloat16*)x;
    a.gate_in = (const __nv_bfloat16*)gate_in;
    a.gate_in_stride = gate_in_stride;
    a.weight = (const __nv_bfloat16*)weight;
    a.style = (const __nv_bfloat16*)style;
    a.style_stride = style_stride;
    a.out = out_bf16;
    a.sf_out = nullptr;
    a.gate_out = (__nv_bfloat16*)gate_out;
    a.d_scale = nullptr;
    a.rows = rows;
    a.dim = dim;
    a.eps = eps;
    cudaStream_t s = (cudaStream_t)stream;
    bool pdl = flags & 1;
    if (x) {
        if (gate_in) {
            if (style) return launch_norm<true, true, true, OUT_BF16>(a, s, pdl);
            return launch_norm<true, true, false, OUT_BF16>(a, s, pdl);
        }
        if (style) return launch_norm<true, false, true, OUT_BF16>(a, s, pdl);
        return launch_norm<true, false, false, OUT_BF16>(a, s, pdl);
    }
    if (style) return launch_norm<false, false, true, OUT_BF16>(a, s, pdl);
    return launch_norm<false, false, false, OUT_BF16>(a, s, pdl);
}

// Same fused norm with an NVFP4 result: packed e2m1 (rows, dim / 2) and block scales in the GEMM's scale-factor
// atoms (zero-filled by the caller once).  The modulated value is rounded to bf16 first, so the result equals
// frt_b200_norm_bf16 followed by frt_b200_quantize_nvfp4 byte for byte.  dim % 16 == 0.  family: 0 / 1.
int frt_b200_norm_nvfp4(void* residual, const void* x, const void* gate_in, long long gate_in_stride,
                        const void* weight, const void* style, long long style_stride, void* out_packed,
                        void* out_sf, void* gate_out, int rows, int dim, float eps, int family, int flags,
                        void* stream) {
    if (!residual || !out_packed || !out_sf) return FRT_ERR_INVALID;
    if (gate_in && !x) return FRT_ERR_INVALID;
    if (family != 0 && family != 1) return FRT_ERR_INVALID;
    if (dim % 16) return FRT_ERR_UNSUPPORTED;
    if (misaligned16(residual) || misaligned16(x) || misaligned16(gate_in) || misaligned16(weight) ||
        misaligned16(style) || misaligned16(gate_out) || (reinterpret_cast<uintptr_t>(out_packed) & 3))
        return FRT_ERR_INVALID;
    if ((gate_in_stride & 7) || (style_stride & 7)) return FRT_ERR_INVALID;
    NormArgs a;
    a.residual = (__nv_bfloat16*)residual;
    a.x = (const __nv_bfloat16*)x;
    a.gate_in = (const __nv_bfloat16*)gate_in;
    a.gate_in_stride = gate_in_stride;
    a.weight = (const __nv_bfloat16*)weight;
    a.style = (const __nv_bfloat16*)style;
    a.style_stride = style_stride;
    a.out = out_packed;
    a.sf_out = (uint8_t*)out_sf;
    a.gate_out = (__nv_bfloat16*)gate_out;
    a.d_scale = nullptr;
    a.rows = rows;
    a.dim = dim;
    a.eps = eps;
    cudaStream_t s = (cudaStream_t)stream;
    if (family == 0) return dispatch_norm_nvfp4<OUT_NVFP4_A>(a, x != nullptr, gate_in != nullptr, style != nullptr, s, flags & 1);
    return dispatch_norm_nvfp4<OUT_NVFP4_B>(a, x != nullptr, gate_in != nullptr, style != nullptr, s, flags & 1);
}

}  // extern "C"
