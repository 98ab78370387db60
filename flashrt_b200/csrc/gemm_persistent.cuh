// Large-M FP8 GEMM as a persistent kernel: one CTA per SM walks a static list of 128 x BN output tiles.
//
// Included by gemm_fp8.cu inside namespace frt (GemmParams, tensor-map cache, status word).
//
// Why: with one tile per CTA the prologue (barriers, TMEM allocation, first TMA round trip) and the epilogue
// (TMEM -> registers -> global) of every tile are exposed; at K = 1024 they cost more than the MMAs.  Here
//   * the TMA producer runs ahead across tile boundaries (the shared-memory ring never drains),
//   * two accumulators live in TMEM (2 x BN columns): the MMA warp fills one while eight epilogue warps drain
//     the other, so the epilogue -- including the bias + GELU + FP8 form -- hides behind the next mainloop,
//   * the tile list is walked in groups of m-tiles (TileOrder), so that the CTAs of a wave share operand rows in L2.
// Warps: 0 TMA producer, 1 MMA issuer (+ TMEM owner), 2..9 epilogue (lane quadrant = warp % 4, column half =
// (warp - 2) / 4).  Every wait is bounded by the kernel deadline; on expiry the status word is set and all roles
// leave their loops.
#pragma once

// EPI_P_BIAS_GELU_FAST_FP8: the same epilogue with the GELU through the hardware tanh -- a template value, not a run-time
// flag: a select inside the unrolled loop over a thread's values costs as much as the arithmetic it chooses between
// EPI_P_GEGLU_FP8 (CTA pairs only): the tile's columns are 128 gate features and the 128 up features that belong to them.
// EPI_P_ROPE (NVFP4 CTA pairs): the QKV projection's RoPE + split + KV append, as EPI_ROPE_SPLIT of the small-M kernel.
enum { EPI_P_BF16 = 0, EPI_P_BIAS_GELU_FP8 = 1, EPI_P_BIAS_GELU_FAST_FP8 = 2, EPI_P_GEGLU_FP8 = 3, EPI_P_ROPE = 4 };

// tanh-form GELU with explicitly rounded fp32 operations, the same sequence as bias_gelu_fp8_kernel
// (csrc/quantize/bias_gelu_quantize_fp8.cu:24-49 in the reference)
__device__ __forceinline__ float gelu_tanh_form_rn(float x) {
    const float x3 = __fmul_rn(__fmul_rn(x, x), x);
    const float u = __fmul_rn(0.7978845608f, __fmaf_rn(0.044715f, x3, x));
    const float e = det_expf(__fmul_rn(2.0f, u));
    const float th = __fsub_rn(1.0f, __fdiv_rn(2.0f, __fadd_rn(1.0f, e)));
    return __fmul_rn(__fmul_rn(0.5f, x), __fadd_rn(1.0f, th));
}

// Order of the output tiles: groups of `gm` m-tiles, inside a group m fastest.  The CTAs of a wave then cover gm m-tiles x
// (wave / gm) n-tiles, and the operand rows they read between them are the fewest when the two extents are alike in bytes.
// (With all m-tiles of one n-tile in a row, the default before, a wave of 148 CTAs reads 148 activation tiles and one weight
// tile: at 40560 x 3072 x 14336 the activations then come from HBM once per n-tile, 7 GB instead of 1.6.)
struct TileOrder {
    int gm, m_tiles, n_tiles;
    __device__ __forceinline__ void at(int t, int& m, int& n) const {
        const int per = gm * n_tiles;
        const int g = t / per, r = t - g * per;
        const int left = m_tiles - g * gm;
        const int h = left < gm ? left : gm;
        n = r / h;
        m = g * gm + (r - n * h);
    }
};
// group height for tiles of tm x tn rows on `workers` CTAs (or pairs): tm * gm = tn * workers / gm
static int tile_group(int m_tiles, int n_tiles, int tm, int tn, int workers) {
    if ((long long)m_tiles * n_tiles <= workers) return m_tiles;
    int gm = 1;
    while ((long long)(gm + 1) * (gm + 1) * tm <= (long long)tn * workers) ++gm;
    return gm < m_tiles ? gm : m_tiles;
}

// The line form of the bf16 epilogue.  BIAS is a template value: a per-value choice between alpha * acc and alpha * acc + bias,
// with the bias unpacked either way, made this loop 450 instructions per 64 columns instead of 120 (0.5 us per 128 x 128 tile
// where nothing hides it).
template <int NC, bool BIAS>
__device__ __forceinline__ void epilogue_bf16_lines(const GemmParams& p, uint32_t t_src, int m_base, int n0, uint8_t* stg,
                                                    float alpha, uint32_t release) {
    const int lane = threadIdx.x & 31;
    const uint32_t stg_w = tc::smem_u32(stg) + lane * 128, sw = (uint32_t)(lane & 7) << 4;
    const int ch = lane & 7, r0 = lane >> 3;
    const uint32_t stg_r = tc::smem_u32(stg) + r0 * 128;
    const int rows = p.M - m_base - r0;                     // row r0 + 4 i exists while 4 i < rows
#pragma unroll 1
    for (int c = 0; c < NC; c += 64) {
        uint32_t v[64];
        tc::tmem_ld32(t_src + c, v);
        tc::tmem_ld32(t_src + c + 32, v + 32);
        tc::tmem_ld_wait();
        if (NC == 64 && release) {                          // these columns may be overwritten from here on
            tc::tc_fence_before_sync();
            tc::mbar_arrive_cluster(release);
        }
        const int nb = n0 + c;
        // this thread's row: 64 results -> bf16 -> eight 16-byte chunks, chunk index xor (row & 7)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float f[8];
            if (BIAS) {
                uint4 bv = make_uint4(0, 0, 0, 0);
                if (nb + 8 * k + 8 <= p.N) bv = ld_global_v4(p.bias + nb + 8 * k);
                const uint32_t* bw = &bv.x;
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    float b0, b1;
                    unpack_bf16x2(bw[e >> 1], b0, b1);
                    f[e] = scale_bias(__uint_as_float(v[8 * k + e]), alpha, b0, true);
                    f[e + 1] = scale_bias(__uint_as_float(v[8 * k + e + 1]), alpha, b1, true);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = scale_bias(__uint_as_float(v[8 * k + e]), alpha, 0.0f, false);
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stg_w + (((uint32_t)k << 4) ^ sw)),
                         "r"(pack_bf16x2(f[0], f[1])), "r"(pack_bf16x2(f[2], f[3])), "r"(pack_bf16x2(f[4], f[5])),
                         "r"(pack_bf16x2(f[6], f[7]))
                         : "memory");
        }
        __syncwarp();
        // four rows x 128 bytes per instruction
        const bool in = nb + ch * 8 + 8 <= p.N;
        __nv_bfloat16* dst = p.out + (size_t)(m_base + r0) * p.N + nb + ch * 8;
        const size_t step = (size_t)4 * p.N;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint4 o;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                         : "r"(stg_r + i * 512 + ((uint32_t)(ch ^ ((4 * i + r0) & 7)) << 4))
                         : "memory");
            if (in && 4 * i < rows) st_global_v4(dst + i * step, o);
        }
        __syncwarp();
    }
}

// One epilogue warp: its 32 rows x NC columns of a finished accumulator (t_src = tensor-memory address of the warp's lane
// quadrant and first column) -> bf16 (+ bias) or bias + GELU + FP8.  `stg` = 4 KB of this warp: tcgen05.ld delivers "thread
// = row"; through shared memory the store instructions become whole lines (8 threads = 128 bytes of a row) instead of 32
// separate half-sectors.  `lines`: rows and bias are 16-byte aligned; otherwise every thread stores its row directly.
// `release` (bf16, NC = 64): a barrier on which every thread arrives as soon as the accumulator's columns are in registers.
template <int EPI, int NC>
__device__ __forceinline__ void epilogue_rows(const GemmParams& p, uint32_t t_src, int m_base, int n0, uint8_t* stg,
                                              bool lines, float alpha, float inv_os, uint32_t release = 0) {
    const int lane = threadIdx.x & 31;
    const int m = m_base + lane;
    if (EPI == EPI_P_BF16) {
        if (lines) {
            if (p.bias) epilogue_bf16_lines<NC, true>(p, t_src, m_base, n0, stg, alpha, release);
            else epilogue_bf16_lines<NC, false>(p, t_src, m_base, n0, stg, alpha, release);
            return;
        }
#pragma unroll 1
        for (int c = 0; c < NC; c += 32) {
            uint32_t v[32];
            __syncwarp();                                   // tcgen05.ld is the whole warp's; lanes beyond M skip the stores
            tc::tmem_ld32(t_src + c, v);
            tc::tmem_ld_wait();
            if (m >= p.M) continue;
            const int nb = n0 + c;
            __nv_bfloat16* orow = p.out + (size_t)m * p.N + nb;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                if (nb + j + 8 <= p.N && ((reinterpret_cast<uintptr_t>(orow + j) & 15) == 0)) {
                    float f[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        f[e] = scale_bias(__uint_as_float(v[j + e]), alpha,
                                          p.bias ? __bfloat162float(p.bias[nb + j + e]) : 0.0f, p.bias != nullptr);
                    uint4 o;
                    o.x = pack_bf16x2(f[0], f[1]);
                    o.y = pack_bf16x2(f[2], f[3]);
                    o.z = pack_bf16x2(f[4], f[5]);
                    o.w = pack_bf16x2(f[6], f[7]);
                    st_global_v4(orow + j, o);
                } else {
                    for (int e = 0; e < 8; ++e)
                        if (nb + j + e < p.N)
                            orow[j + e] = __float2bfloat16_rn(scale_bias(
                                __uint_as_float(v[j + e]), alpha, p.bias ? __bfloat162float(p.bias[nb + j + e]) : 0.0f,
                                p.bias != nullptr));
                }
            }
        }
        if (release) {
            tc::tc_fence_before_sync();
            tc::mbar_arrive_cluster(release);
        }
        return;
    }
    // bf16(alpha * acc) + bias -> GELU -> e4m3: the rounding points of GEMM -> bias_gelu_quantize.  N % 8 == 0; a row of NC
    // bytes is staged as NC / 16 chunks of 16, chunk index xor (row & (NC / 16 - 1))
    constexpr int CH = NC / 16;
    const bool hb = p.bias != nullptr;
    const bool bvec = hb && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
#pragma unroll 1
    for (int c = 0; c < NC; c += 32) {
        uint32_t v[32];
        __syncwarp();                                       // the lanes part where they store their own rows
        tc::tmem_ld32(t_src + c, v);
        tc::tmem_ld_wait();
        const int nb = n0 + c;
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            float g[8], bj[8];
            const bool in = nb + j + 8 <= p.N;
            // 8 bias values with one load when they are 16-byte aligned (nb + j is a multiple of 8)
            if (bvec && in) {
                const uint4 bv = ld_global_v4(p.bias + nb + j);
                unpack_bf16x2(bv.x, bj[0], bj[1]);
                unpack_bf16x2(bv.y, bj[2], bj[3]);
                unpack_bf16x2(bv.z, bj[4], bj[5]);
                unpack_bf16x2(bv.w, bj[6], bj[7]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) bj[e] = hb && in ? __bfloat162float(p.bias[nb + j + e]) : 0.0f;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float x = bf16_round(__uint_as_float(v[j + e]) * alpha);
                if (hb) x = __fadd_rn(x, bj[e]);
                g[e] = clamp448(__fmul_rn(EPI == EPI_P_BIAS_GELU_FAST_FP8 ? fast_gelu_tanh(x) : gelu_tanh_form_rn(x), inv_os));
            }
            w[j / 4] = f32x4_to_e4m3x4(g[0], g[1], g[2], g[3]);
            w[j / 4 + 1] = f32x4_to_e4m3x4(g[4], g[5], g[6], g[7]);
            if (!lines && m < p.M && in)
                st_global_v2(p.out8 + (size_t)m * p.N + nb + j, make_uint2(w[j / 4], w[j / 4 + 1]));
        }
        if (lines) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ch = c / 16 + h;
                *reinterpret_cast<uint4*>(stg + lane * NC + ((ch ^ (lane & (CH - 1))) << 4)) =
                    make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
            }
        }
    }
    if (lines) {
        __syncwarp();
        const int ch = lane % CH;
#pragma unroll
        for (int r0 = 0; r0 < 32; r0 += 32 / CH) {
            const int row = r0 + lane / CH;
            const uint4 o = *reinterpret_cast<const uint4*>(stg + row * NC + ((ch ^ (row & (CH - 1))) << 4));
            const int mm = m_base + row, nn = n0 + ch * 16;
            if (mm < p.M && nn + 16 <= p.N) st_global_v4(p.out8 + (size_t)mm * p.N + nn, o);
        }
        __syncwarp();
    }
}

// The same for 32 gate columns (t_gate) and their 32 up columns (t_up): e4m3(gelu_tanh(bf16(gate)) * bf16(up) / scale) at
// features h0 .. h0 + 31 of out8 (M, half), the rounding points of GEMM -> geglu_fp8.  A thread's 32 bytes are one sector.
__device__ __forceinline__ void epilogue_geglu_rows(const GemmParams& p, uint32_t t_gate, uint32_t t_up, int m_base, int h0,
                                                    float alpha, float inv_os) {
    if (m_base >= p.M) return;
    const int m = m_base + (threadIdx.x & 31);
    uint32_t g[32], u[32], w[8];
    __syncwarp();                                           // lanes beyond M skip the stores of the call before
    tc::tmem_ld32(t_gate, g);
    tc::tmem_ld32(t_up, u);
    tc::tmem_ld_wait();
    const uint64_t al2 = f32x2(alpha, alpha), io2 = f32x2(inv_os, inv_os);
    // rows beyond M hold zeros, and a zero takes the activation's slow path (541 rows: 48 us a launch with it)
    if (m >= p.M) {
#pragma unroll
        for (int j = 0; j < 32; ++j) g[j] = 0x3f800000u;
    }
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            auto rounded = [&](const uint32_t* v) {          // bf16(alpha * v) of two columns
                float v0, v1;
                f32x2_parts(mul_f32x2(f32x2(__uint_as_float(v[0]), __uint_as_float(v[1])), al2), v0, v1);
                return unpack_bf16x2(pack_bf16x2(v0, v1));
            };
            f32x2_parts(mul_f32x2(mul_f32x2(det_gelu_tanh2(rounded(g + j + e)), rounded(u + j + e)), io2), o[e], o[e + 1]);
        }
        w[j / 4] = f32x4_to_e4m3x4(clamp448(o[0]), clamp448(o[1]), clamp448(o[2]), clamp448(o[3]));
    }
    if (m < p.M) {
        uint8_t* dst = p.out8 + (size_t)m * p.half + h0;
        st_global_v4(dst, make_uint4(w[0], w[1], w[2], w[3]));
        st_global_v4(dst + 16, make_uint4(w[4], w[5], w[6], w[7]));
    }
}

// 64 features of the fused q|k|v row of one token per thread: bf16(alpha * acc) rotated (V: copied), the rounding points of
// EPI_ROPE_SPLIT.  `tab`: the token's 64 table values, fetched while the MMAs run (rope_table_rows).
__device__ __forceinline__ int rope_column(const GemmParams& p, int n) {     // feature within its q, k or v part
    return n < p.q_dim ? n : n < p.q_dim + p.k_dim ? n - p.q_dim : n - p.q_dim - p.k_dim;
}
__device__ __forceinline__ void rope_table_rows(const GemmParams& p, int m, int n0, uint4* tab) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int n = n0 + 8 * c;
        tab[c] = make_uint4(0, 0, 0, 0);
        if (m < p.M && n < p.q_dim + p.k_dim)
            tab[c] = ld_global_v4(p.rope + (size_t)m * p.head_dim + rope_column(p, n) % p.head_dim);
    }
}
__device__ __forceinline__ void epilogue_rope_rows(const GemmParams& p, uint32_t t_src, int m, int n0, float alpha, int pos,
                                                   const uint4* tab) {
    uint32_t a[64];
    __syncwarp();                                           // lanes beyond M skip the stores of the call before
    tc::tmem_ld32(t_src, a);
    tc::tmem_ld32(t_src + 32, a + 32);
    tc::tmem_ld_wait();
    if (m >= p.M) return;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int n = n0 + 8 * c;
        if (n >= p.N) break;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = bf16_round(__uint_as_float(a[8 * c + j]) * alpha);
        const bool is_q = n < p.q_dim, is_k = !is_q && n < p.q_dim + p.k_dim;
        const int nr = rope_column(p, n);
        uint4 o;
        if (is_q || is_k) {
            const uint32_t* tw = &tab[c].x;
            uint32_t* ow = &o.x;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float cs, sn;
                unpack_bf16x2(tw[k], cs, sn);
                ow[k] = pack_bf16x2(__fmaf_rn(v[2 * k], cs, -__fmul_rn(v[2 * k + 1], sn)),
                                    __fmaf_rn(v[2 * k + 1], cs, __fmul_rn(v[2 * k], sn)));
            }
        } else {
            o = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        }
        __nv_bfloat16* dst = is_q ? p.outQ + (size_t)m * p.q_dim + nr
                                  : (is_k ? p.outK + (size_t)(pos + m) * p.k_dim + nr : p.outV + (size_t)(pos + m) * p.v_dim + nr);
        st_global_v4(dst, o);
    }
}

// whole-line stores are possible: 16-byte rows and bias
template <int EPI>
__device__ __forceinline__ bool epilogue_lines(const GemmParams& p) {
    if (EPI == EPI_P_BF16)
        return (p.N % 8) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 &&
               (!p.bias || (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0);
    return (p.N % 16) == 0 && (reinterpret_cast<uintptr_t>(p.out8) & 15) == 0;
}

template <int BN>
struct PGemmCfg {
    static constexpr int L_BYTES = 128 * 128;
    static constexpr int C_BYTES = BN * 128;
    static constexpr int STAGE_BYTES = L_BYTES + C_BYTES;
    static constexpr int MAX_STAGES = (227 * 1024 - 2048) / STAGE_BYTES;
    static constexpr int STAGES = MAX_STAGES > 6 ? 6 : MAX_STAGES;
    // bf16 epilogue staging: every epilogue warp owns 32 rows x 128 bytes, through which its 32 x 64 block of results is
    // turned from "thread = row" (what tcgen05.ld gives) into "8 threads = one 128-byte line" for the global store
    static constexpr int EPI_STAGE_BYTES = 8 * 32 * 128;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + EPI_STAGE_BYTES;
    static constexpr int TMEM_COLS = 2 * BN;          // BN in {128, 256}
    static constexpr int EPI_THREADS = 256;
};

template <int BN, int EPI>
__global__ void __launch_bounds__(320, 1)
gemm_fp8_persistent_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                           GemmParams p) {
    using Cfg = PGemmCfg<BN>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;      // [2]
    uint64_t* acc_empty = acc_full + 2;       // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const uint64_t deadline = tc::global_timer_ns() + FRT_KERNEL_DEADLINE_NS;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int m_tiles = (p.M + 127) / 128;
    const int n_tiles = (p.N + BN - 1) / BN;
    const int total = m_tiles * n_tiles;
    const int kbt = p.kb_total;
    const TileOrder order = {p.tile_gm, m_tiles, n_tiles};

    // The producer warp sets the barriers up and goes straight to its first copies; the other warps meet it at barrier 2
    // (where it only arrives): tensor-memory allocation and the meeting are off the way to the first byte.
    uint32_t tmem = 0;
    if (warp == 0) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&tmA);
            tc::tma_prefetch_desc(&tmW);
            for (int s = 0; s < STAGES; ++s) {
                tc::mbar_init(&full[s], 1);
                tc::mbar_init(&empty[s], 1);
            }
            for (int i = 0; i < 2; ++i) {
                tc::mbar_init(&acc_full[i], 1);
                tc::mbar_init(&acc_empty[i], Cfg::EPI_THREADS);
            }
            *abort_flag = 0;
            tc::mbar_fence_init();
        }
        __syncwarp();
        asm volatile("barrier.cta.arrive 2, 320;" ::: "memory");
    } else {
        if (warp == 1) {
            tc::tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
            tc::tmem_relinquish();
        }
        tc::tc_fence_before_sync();
        asm volatile("barrier.cta.sync 2, 320;" ::: "memory");
        tc::tc_fence_after_sync();
        tmem = *tmem_slot;
    }

    pdl_launch_dependents();

    if (warp == 0) {
        // ---------------- TMA producer (whole warp, see warp_wait): runs ahead over tile boundaries
        pdl_wait();
        const uint32_t ring = tc::smem_u32(smem), full_a = tc::smem_u32(full), empty_a = tc::smem_u32(empty);
        int s = 0;                    // ring position; no division on this path
        uint32_t ph = 1;              // parity that an empty slot has completed (a fresh barrier passes parity 1)
        bool ready = true;
        for (int t = blockIdx.x; t < total; t += gridDim.x) {
            int mt, nt;
            order.at(t, mt, nt);
            const int m0 = mt * 128, n0 = nt * BN;
            for (int kb = 0; kb < kbt; ++kb) {
                if (!tc::warp_wait(empty_a + 8 * s, ph, ready, deadline, abort_flag)) {
                    if (lane == 0 && !*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_PRODUCER | (blockIdx.x << 8));
                    *abort_flag = 1;
                    t = total;
                    break;
                }
                const uint32_t dst = ring + s * Cfg::STAGE_BYTES, bar = full_a + 8 * s;
                if (++s == STAGES) { s = 0; ph ^= 1; }
                ready = tc::mbar_test(empty_a + 8 * s, ph);
                if (tc::elect_one()) {
                    tc::mbar_arrive_expect_tx(bar, Cfg::STAGE_BYTES);
                    tc::tma_load_2d(dst, &tmA, bar, kb * 128, m0);
                    if (p.w_kn) {      // (K, N) weights: one 128 x 128-byte box per 128 output features
#pragma unroll
                        for (int j = 0; j < BN / 128; ++j)
                            tc::tma_load_2d(dst + Cfg::L_BYTES + j * 16384, &tmW, bar, n0 + j * 128, kb * 128);
                    } else {
                        tc::tma_load_2d(dst + Cfg::L_BYTES, &tmW, bar, kb * 128, n0);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (whole warp): accumulator i & 1 for the CTA's i-th tile
        const bool w_kn = p.w_kn;
        const uint32_t idesc = tc::make_idesc(0, 0, 0, 0, 128, BN) | (w_kn ? (1u << 16) : 0u);
        const uint64_t dL0 = tc::make_desc_kmajor_sw128(tc::smem_u32(smem));
        const uint64_t dC0 = w_kn ? tc::make_desc_mnmajor_sw128(tc::smem_u32(smem + Cfg::L_BYTES), 16384)
                                  : tc::make_desc_kmajor_sw128(tc::smem_u32(smem + Cfg::L_BYTES));
        const uint64_t cstep = w_kn ? (uint64_t)((32 * 128) >> 4) : 2u;
        const uint32_t full_a = tc::smem_u32(full), empty_a = tc::smem_u32(empty);
        const uint32_t accF_a = tc::smem_u32(acc_full), accE_a = tc::smem_u32(acc_empty);
        int s = 0, i = 0;
        uint32_t ph = 0;
        bool ready = false, failed = false;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++i) {
            const int buf = i & 1;
            if (!tc::warp_wait(accE_a + 8 * buf, (uint32_t)(((i >> 1) - 1) & 1), i < 2, deadline, abort_flag)) {
                if (lane == 0 && !*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_MMA | (blockIdx.x << 8));
                *abort_flag = 1;
                break;
            }
            tc::tc_fence_after_sync();
            const uint32_t d_tm = tmem + buf * BN;
            for (int kb = 0; kb < kbt; ++kb) {
                if (!tc::warp_wait(full_a + 8 * s, ph, ready, deadline, abort_flag)) {
                    if (lane == 0 && !*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_MMA | (blockIdx.x << 8));
                    *abort_flag = 1;
                    failed = true;
                    break;
                }
                tc::tc_fence_after_sync();
                const uint64_t so = (uint64_t)(s * (Cfg::STAGE_BYTES >> 4));
                const uint32_t done = empty_a + 8 * s;
                if (++s == STAGES) { s = 0; ph ^= 1; }
                ready = tc::mbar_test(full_a + 8 * s, ph);
                if (tc::elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tc::mma_f8(d_tm, dL0 + so + 2 * k, dC0 + so + cstep * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc::mma_commit(done);
                    if (kb == kbt - 1) tc::mma_commit(accF_a + 8 * buf);
                }
            }
            if (failed) break;
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: eight warps drain one accumulator while the other one fills
        pdl_wait();
        const int q = warp & 3;                         // TMEM lane quadrant this warp may access
        const int half = (warp - 2) >> 2;               // which half of the BN columns
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        float alpha = p.alpha_host;
        if (p.sa) alpha *= *p.sa;
        if (p.sb) alpha *= *p.sb;
        const float inv_os = (EPI != EPI_P_BF16) ? __fdiv_rn(1.0f, *p.out_scale) : 0.0f;
        const bool lines = epilogue_lines<EPI>(p);
        uint8_t* stg = smem + STAGES * Cfg::STAGE_BYTES + 256 + (warp - 2) * (32 * 128);
        int i = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++i) {
            const int buf = i & 1;
            const bool ok = tc::mbar_wait_until(&acc_full[buf], (uint32_t)((i >> 1) & 1), deadline, abort_flag);
            if (!__all_sync(0xffffffffu, ok)) {          // leave as a whole warp: tcgen05.ld is warp-collective
                if (!*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_EPILOGUE | (blockIdx.x << 8));
                *abort_flag = 1;
                break;
            }
            tc::tc_fence_after_sync();
            int mt, nt;
            order.at(t, mt, nt);
            epilogue_rows<EPI, BN / 2>(p, tmem + buf * BN + half * (BN / 2) + lane_off, mt * 128 + q * 32,
                                       nt * BN + half * (BN / 2), stg, lines, alpha, inv_os);
            tc::tc_fence_before_sync();
            tc::mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, Cfg::TMEM_COLS);
}

template <int BN, int EPI>
static int launch_gemm_persistent(const void* A, const void* W, GemmParams p, int K, cudaStream_t stream) {
    using Cfg = PGemmCfg<BN>;
    static PerDeviceOnce attr_once;
    int attr_dev = 0;
    const int sms = device_sm_count();
    if (attr_once.need(attr_dev)) {
        cudaError_t e = cudaFuncSetAttribute(gemm_fp8_persistent_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             Cfg::SMEM_BYTES);
        if (e != cudaSuccess) return FRT_CUDA_ERR(e);
        attr_once.set(attr_dev);
    }
    CUtensorMap tmA, tmW;
    int rc = get_tmap_2d_u8(&tmA, A, (uint64_t)p.M, (uint64_t)K, (uint64_t)K, 128);
    if (rc) return rc;
    rc = p.w_kn ? get_tmap_2d_u8(&tmW, W, (uint64_t)K, (uint64_t)p.N, (uint64_t)p.N, 128)
                : get_tmap_2d_u8(&tmW, W, (uint64_t)p.N, (uint64_t)K, (uint64_t)K, BN);
    if (rc) return rc;
    const int m_tiles = (p.M + 127) / 128, n_tiles = (p.N + BN - 1) / BN, total = m_tiles * n_tiles;
    p.tile_gm = tile_group(m_tiles, n_tiles, 128, BN, sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(total < sms ? total : sms);
    cfg.blockDim = dim3(320);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;                   // nothing global is read before the wait
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_fp8_persistent_kernel<BN, EPI>, tmA, tmW, p);
    return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
}
