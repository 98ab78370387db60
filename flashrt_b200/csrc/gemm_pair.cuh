// Large-M FP8 GEMM with one 256 x 256 output tile per CTA PAIR (tcgen05 cta_group::2), persistent.
//
// Included by gemm_fp8.cu inside namespace frt (GemmParams, tensor-map cache, status word, gemm_persistent.cuh).
//
// Why: with one CTA per 128 x 256 tile every MMA of 128 x 256 x 32 reads 4 KB of A and 8 KB of B from that CTA's
// shared memory -- 96 bytes per clock of the 128 the SM can deliver, and the K = 1024 shapes stall on it.  A pair
// of CTAs (a cluster of two) computes 256 x 256: each CTA stages ITS 128 rows of A and ITS 128 of the 256 weight
// rows (16 KB + 16 KB per k-block instead of 16 + 32), the leader CTA issues one tcgen05.mma.cta_group::2 that
// reads both CTAs' shared memory, and each CTA receives its 128 rows x 256 columns of the result in its own
// tensor memory.  Same bytes from L2 per flop as two independent 128 x 256 tiles sharing a weight tile, but two
// thirds of the shared-memory operand traffic per SM.
//
// Protocol (rank 0 = leader):
//   * both producers wait for their own empty[s], the leader posts the byte count of BOTH CTAs on its full[s], both
//     issue their TMA loads (cta_group::2 form, no multi-destination copy) signalling the LEADER's full[s];
//   * the leader's MMA thread waits for full[s], issues four MMAs (K = 32 each) and commits to empty[s] of both CTAs,
//     likewise for acc_full[buf];
//   * eight epilogue warps per CTA drain that CTA's accumulator and arrive on the leader's acc_empty[buf]
//     (one arrival per epilogue thread of both), which the leader's MMA thread waits for before it reuses the buffer.
// Tensor memory is allocated and freed with the cta_group::2 forms by the same warp of both CTAs.  Every wait is
// bounded by the kernel deadline; the CTAs meet at a cluster barrier before either leaves.
#pragma once

//
// NVFP4 (FP4 = true): the same protocol with k-blocks of 256 packed e2m1 elements (128 bytes a row) and, behind the operand
// tiles of a stage, the block scales: the CTA's own 128 rows of A (2 KB) and ALL the tile's columns (2 KB per 128; 192 columns
// touch two atom rows wherever they start, at row 0 or 64 of the first), since each SM multiplies its 128 rows by every
// column.  They go to tensor memory with tcgen05.cp in front of the k-block's MMAs.  What bounds this product is the operand
// traffic from L2: a 128 x 128 tile per CTA takes 36 KB per 270 clocks of math, a pair of 256 x 256 38 KB per 540.
// 256 columns: two accumulators and the 48 scale columns are more than the 512 of tensor memory, so the accumulators share
// 64 columns (0..255 and 192..447).  The warps that hold the shared columns read them first and release them at once; the
// MMAs of the next tile wait for that one read (about 0.3 us per tile) and not for the finish.
template <int BN, bool FP4 = false>                       // columns of the pair's tile (BN / 2 weight rows per CTA)
struct GemmPairCfg {
    static constexpr int A_BYTES = 128 * 128;
    static constexpr int B_BYTES = BN / 2 * 128;
    static constexpr int SFA_BYTES = FP4 ? 2048 : 0;
    static constexpr int SFB_ROWS = (BN + 127) / 128;       // 128-row atom rows of the columns' scales
    static constexpr int SFB_BYTES = FP4 ? SFB_ROWS * 2048 : 0;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES;   // per CTA
    static constexpr int STAGES = FP4 ? (BN >= 192 ? 5 : 6) : BN >= 192 ? 6 : 8;
    static constexpr int EPI_STAGE_BYTES = 8 * 32 * 128;    // line staging of the eight epilogue warps
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + EPI_STAGE_BYTES;
    static constexpr int TMEM_COLS = BN == 128 && !FP4 ? 256 : 512;  // two accumulators (and the scales)
    static constexpr bool OVERLAP = FP4 && BN == 256;
    static constexpr int ACC_STRIDE = OVERLAP ? 192 : BN;   // columns from one accumulator to the other
    static constexpr int SF_COL = ACC_STRIDE + BN;          // scales of A: 4 columns per K = 64; of W: 4 per atom row
};
// epilogue threads per CTA: the GeGLU finish is a chain of 30 dependent instructions per value, which sixteen warps hide
// where eight do not
template <int EPI>
constexpr int pair_epi_threads() { return EPI == EPI_P_GEGLU_FP8 ? 512 : 256; }

namespace tc {
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {   // same warp of both CTAs
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// tiled load whose completion bytes are posted on a barrier given as a shared::cluster address (the leader's)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int x,
                                                 int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_dst), "l"(m), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}
// D[tmem of both CTAs] (+)= A[both CTAs' smem] . B[both CTAs' smem]; issued by one thread of the leader CTA
__device__ __forceinline__ void mma_f8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z)
        : "memory");
}
// all MMAs issued so far by this thread -> one arrival on the barrier at this shared-memory offset in both CTAs of the pair
__device__ __forceinline__ void mma_commit_both(uint32_t bar_addr) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar_addr),
        "h"((uint16_t)3)
        : "memory");
}
}  // namespace tc

// One of the S arrivals at a (tile, epilogue warp) counter, by one lane: the number of arrivals before it.  The S-th takes the
// counter back to zero in the same operation, so a launch leaves all of them at zero as long as every unit arrives once --
// a warp whose wait gave up arrives for its remaining units too (the sums it spoils are reported by the status word).
__device__ __forceinline__ int split_k_arrive(const GemmParams& p, int unit, int S, int slot) {
    return (int)atomicInc(p.split_cnt + (unit / S) * 16 + slot, (unsigned)(S - 1));
}

// Split K: an epilogue warp's 32 rows x NC columns of one split.  It leaves its partial in the workspace ([unit][warp][NC / 4]
// [lane][4] floats: 512 bytes per store), then counts itself in; the last of the tile's S warps adds the partials in split
// order, its own from tensor memory, and puts the sum back there for the finish.  Nobody waits.  False: not the last.
template <int NC>
__device__ __forceinline__ bool split_k_sum(const GemmParams& p, uint32_t t_src, int unit, int S, int slot) {
    const int lane = threadIdx.x & 31;
    const int mine = unit % S, first = unit - mine;
    auto base = [&](int u) { return p.split_ws + ((size_t)u * 16 + slot) * (32 * NC) + lane * 4; };
    float* out = base(unit);
#pragma unroll 1
    for (int c = 0; c < NC; c += 32) {
        uint32_t v[32];
        tc::tmem_ld32(t_src + c, v);
        tc::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
            __stcg(reinterpret_cast<uint4*>(out + (c + j) * 32), make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]));
    }
    __threadfence();
    __syncwarp();
    int seen = 0;
    if (lane == 0) seen = split_k_arrive(p, unit, S, slot);
    seen = __shfl_sync(0xffffffffu, seen, 0);
    if (seen != S - 1) return false;
    __threadfence();
#pragma unroll 1
    for (int c = 0; c < NC; c += 32) {
        uint32_t v[32];
        float a[32];
        tc::tmem_ld32(t_src + c, v);
        tc::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) a[j] = 0.0f;
        for (int s = 0; s < S; ++s) {
            if (s == mine) {
#pragma unroll
                for (int j = 0; j < 32; ++j) a[j] += __uint_as_float(v[j]);
            } else {
                const float* in = base(first + s);
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 x = __ldcg(reinterpret_cast<const float4*>(in + (c + j) * 32));
                    a[j] += x.x; a[j + 1] += x.y; a[j + 2] += x.z; a[j + 3] += x.w;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(a[j]);
        tc::tmem_st32(t_src + c, v);
    }
    tc::tmem_st_wait();
    return true;
}

// Maps of the scale atoms (256 bytes of launch parameters): the NVFP4 form's alone.
template <bool FP4>
struct PairScaleMaps {};
template <>
struct PairScaleMaps<true> { CUtensorMap a, w; };

template <int BN, int EPI, bool SPLIT = false, bool FP4 = false>
__global__ void __launch_bounds__(64 + pair_epi_threads<EPI>(), 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, GemmParams p,
                     const __grid_constant__ PairScaleMaps<FP4> sfm) {
    static_assert(BN == 128 || BN == 192 || BN == 256, "tile widths");
    static_assert(!SPLIT || BN == 256, "split K: 256 x 256 tiles");
    static_assert(EPI != EPI_P_GEGLU_FP8 || BN == 256, "GeGLU: 128 gate and 128 up columns");
    static_assert(!FP4 || (!SPLIT && (EPI == EPI_P_BF16 || (EPI == EPI_P_ROPE && BN == 128))), "forms of the NVFP4 product");
    static_assert(EPI != EPI_P_ROPE || FP4, "RoPE finish: NVFP4");
    using Cfg = GemmPairCfg<BN, FP4>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);   // used in the leader only
    uint64_t* empty = full + STAGES;          // one per CTA: the leader's commits arrive on both
    uint64_t* acc_full = empty + STAGES;      // [2] one per CTA
    uint64_t* acc_empty = acc_full + 2;       // [2] used in the leader only
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const uint64_t deadline = tc::global_timer_ns() + FRT_KERNEL_DEADLINE_NS;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_ctarank();          // 0 = leader
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int m_tiles = (p.M + 255) / 256;
    const int n_tiles = (p.N + BN - 1) / BN;
    // SPLIT: a unit is (tile, K split), the splits of a tile next to one another and all of them resident at once
    const int S = SPLIT ? p.ksplits : 1;
    const int total = m_tiles * n_tiles * S;
    const TileOrder order = {p.tile_gm, m_tiles, n_tiles};
    auto k_begin = [&](int t) { return SPLIT ? (int)((long long)p.kb_total * (t % S) / S) : 0; };
    auto k_end = [&](int t) { return SPLIT ? (int)((long long)p.kb_total * (t % S + 1) / S) : p.kb_total; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 2 * pair_epi_threads<EPI>());
        }
        *abort_flag = 0;
        tc::mbar_fence_init();
        tc::tma_prefetch_desc(&tmA);
        tc::tma_prefetch_desc(&tmW);
        if constexpr (FP4) {
            tc::tma_prefetch_desc(&sfm.a);
            tc::tma_prefetch_desc(&sfm.w);
        }
    }
    if (warp == 1) {
        tc::tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
        tc::tmem_relinquish_pair();
    }
    tc::tc_fence_before_sync();
    tc::cluster_sync_all();                    // both CTAs' barriers exist before anything signals across
    tc::tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    pdl_launch_dependents();

    // a k-block of this CTA's activation rows / of its weight rows, with their scales
    auto load_rows = [&](uint32_t dst, uint32_t bar, int kb, int m0) {
        tc::tma_load_2d_pair(dst, &tmA, bar, kb * 128, m0);
        if constexpr (FP4) tc::tma_load_2d_pair(dst + Cfg::A_BYTES + Cfg::B_BYTES, &sfm.a, bar, kb * 256, m0 / 128);
    };
    auto load_weights = [&](uint32_t dst, uint32_t bar, int kb, int n0, int sf_row) {
        tc::tma_load_2d_pair(dst + Cfg::A_BYTES, &tmW, bar, kb * 128, n0);
        if constexpr (FP4)
            tc::tma_load_2d_pair(dst + Cfg::A_BYTES + Cfg::B_BYTES + Cfg::SFA_BYTES, &sfm.w, bar, kb * 256, sf_row);
    };
    auto weight_row = [&](int nt) {          // GeGLU: the leader stages the gate rows of the tile, its peer the up rows
        return EPI == EPI_P_GEGLU_FP8 ? nt * (BN / 2) + (int)rank * p.half : nt * BN + (int)rank * (BN / 2);
    };

    if (warp == 0) {
        // ---------------- TMA producer (whole warp, see warp_wait; both CTAs): its half of A and of the weight rows, bytes posted at the leader
        // Settled weights (p.early): the pair's first ring of weight tiles is fetched before the wait for the kernel in front.
        // Apart from the loop below: its body with one more test and the weights in front of the rows made every product of
        // many k-blocks 1.5 % slower (2048 x 3072 x 3072 16.3 -> 16.5 us, 8192 x 3072 x 3072 59.7 -> 60.6).
        const uint32_t ring = tc::smem_u32(smem), empty_a = tc::smem_u32(empty), full_a = tc::smem_u32(full);
        const uint32_t lead_full = tc::dsmem_map(full_a, 0);
        int ahead = 0, mt, nt;        // k-blocks of the first tile whose weights are on their way
        if (p.early && pair < total) {
            order.at(SPLIT ? pair / S : pair, mt, nt);
            const int kb0 = k_begin(pair), n = k_end(pair) - kb0;
            ahead = n < STAGES ? n : STAGES;
            if (tc::elect_one())
                for (int s = 0; s < ahead; ++s) {
                    if (rank == 0) tc::mbar_arrive_expect_tx(full_a + 8 * s, 2 * Cfg::STAGE_BYTES);
                    load_weights(ring + s * Cfg::STAGE_BYTES, lead_full + 8 * s, kb0 + s, weight_row(nt), nt * BN / 128);
                }
        }
        pdl_wait();
        if (ahead > 0 && tc::elect_one())
            for (int s = 0; s < ahead; ++s)
                load_rows(ring + s * Cfg::STAGE_BYTES, lead_full + 8 * s, k_begin(pair) + s, mt * 256 + (int)rank * 128);
        int s = ahead % STAGES;
        uint32_t ph = ahead < STAGES;   // parity that an empty slot has completed (a fresh barrier passes parity 1)
        bool ready = ahead < STAGES;
        for (int t = pair; t < total; t += npairs) {
            order.at(SPLIT ? t / S : t, mt, nt);
            const int m0 = mt * 256 + (int)rank * 128, n0 = weight_row(nt), sf_row = nt * BN / 128;
            const int kb1 = k_end(t);
            for (int kb = k_begin(t) + (t == pair ? ahead : 0); kb < kb1; ++kb) {
                if (!tc::warp_wait(empty_a + 8 * s, ph, ready, deadline, abort_flag)) {
                    if (lane == 0 && !*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_PRODUCER | (blockIdx.x << 8));
                    *abort_flag = 1;
                    t = total;
                    break;
                }
                const uint32_t dst = ring + s * Cfg::STAGE_BYTES, bar = lead_full + 8 * s;
                const uint32_t own = full_a + 8 * s;
                if (++s == STAGES) { s = 0; ph ^= 1; }
                ready = tc::mbar_test(empty_a + 8 * s, ph);
                if (tc::elect_one()) {
                    if (rank == 0) tc::mbar_arrive_expect_tx(own, 2 * Cfg::STAGE_BYTES);
                    load_rows(dst, bar, kb, m0);
                    load_weights(dst, bar, kb, n0, sf_row);
                }
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ---------------- MMA issuer (whole warp, leader only): accumulator i & 1 for the pair's i-th tile
        constexpr uint32_t idesc = FP4 ? tc::make_idesc_nvfp4(256, BN) : tc::make_idesc(0, 0, 0, 0, 256, BN);
        const uint32_t sf0 = tc::smem_u32(smem + Cfg::A_BYTES + Cfg::B_BYTES);
        const uint32_t tmem_sfa = tmem + Cfg::SF_COL, tmem_sfw = tmem_sfa + 16;
        const uint64_t dA0 = tc::make_desc_kmajor_sw128(tc::smem_u32(smem));
        const uint64_t dB0 = tc::make_desc_kmajor_sw128(tc::smem_u32(smem + Cfg::A_BYTES));
        const uint32_t full_a = tc::smem_u32(full), empty_a = tc::smem_u32(empty);
        int s = 0, i = 0;
        uint32_t ph = 0;
        const uint32_t accF_a = tc::smem_u32(acc_full), accE_a = tc::smem_u32(acc_empty);
        bool ready = false, failed = false;
        for (int t = pair; t < total; t += npairs, ++i) {
            const int buf = i & 1;
            // this accumulator's tile before the last one is drained; with shared columns: those of the last tile are read
            const bool free_acc = Cfg::OVERLAP
                ? tc::warp_wait(accE_a + 8 * (buf ^ 1), (uint32_t)(((i - 1) >> 1) & 1), i < 1, deadline, abort_flag)
                : tc::warp_wait(accE_a + 8 * buf, (uint32_t)(((i >> 1) - 1) & 1), i < 2, deadline, abort_flag);
            if (!free_acc) {
                if (lane == 0 && !*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_MMA | (blockIdx.x << 8));
                *abort_flag = 1;
                break;
            }
            tc::tc_fence_after_sync();
            const uint32_t d_tm = tmem + buf * Cfg::ACC_STRIDE;
            // the tile's first column is row 0 or (192-wide tiles) row 64 of its first scale atom: two columns further on
            uint32_t sfw_tm = tmem_sfw;
            if constexpr (FP4 && BN == 192) {
                int mt, nt;
                order.at(t, mt, nt);
                sfw_tm += (uint32_t)(nt & 1) * 2;
            }
            const int kb0 = k_begin(t), kb1 = k_end(t);
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!tc::warp_wait(full_a + 8 * s, ph, ready, deadline, abort_flag)) {
                    if (lane == 0 && !*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_MMA | (blockIdx.x << 8));
                    *abort_flag = 1;
                    failed = true;
                    break;
                }
                tc::tc_fence_after_sync();
                const uint64_t so = (uint64_t)(s * (Cfg::STAGE_BYTES >> 4));
                const uint32_t sf = sf0 + (uint32_t)(s * Cfg::STAGE_BYTES), done = empty_a + 8 * s;
                if (++s == STAGES) { s = 0; ph ^= 1; }
                ready = tc::mbar_test(full_a + 8 * s, ph);
                if (tc::elect_one()) {
                    if constexpr (FP4) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            tc::tmem_cp_sf_atom_pair(tmem_sfa + 4 * k, sf + 512 * k);
#pragma unroll
                            for (int j = 0; j < Cfg::SFB_ROWS; ++j)
                                tc::tmem_cp_sf_atom_pair(tmem_sfw + (k * Cfg::SFB_ROWS + j) * 4,
                                                         sf + Cfg::SFA_BYTES + j * 2048 + 512 * k);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tc::mma_nvfp4_pair(d_tm, dA0 + so + 2 * k, dB0 + so + 2 * k, idesc, tmem_sfa + 4 * k,
                                               sfw_tm + k * Cfg::SFB_ROWS * 4, (kb > kb0 || k > 0) ? 1u : 0u);
                    } else
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tc::mma_f8_pair(d_tm, dA0 + so + 2 * k, dB0 + so + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
                    tc::mma_commit_both(done);
                    if (kb == kb1 - 1) tc::mma_commit_both(accF_a + 8 * buf);
                }
            }
            if (failed) break;
        }
    } else if (warp >= 2) {
        // ---------------- epilogue (both CTAs): this CTA's 128 rows x 256 columns
        pdl_wait();
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;                 // column half (GeGLU: quarter) of this warp
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        float alpha = p.alpha_host;
        if (p.sa) alpha *= *p.sa;
        if (p.sb) alpha *= *p.sb;
        const float inv_os = EPI != EPI_P_BF16 && EPI != EPI_P_ROPE ? __fdiv_rn(1.0f, *p.out_scale) : 0.0f;
        const bool lines = epilogue_lines<EPI>(p);
        const int pos = EPI == EPI_P_ROPE && p.devpos ? *p.devpos : 0;
        uint8_t* stg = smem + STAGES * Cfg::STAGE_BYTES + 256 + (warp - 2) * (32 * 128);
        int i = 0;
        for (int t = pair; t < total; t += npairs, ++i) {
            const int buf = i & 1;
            uint4 tab[EPI == EPI_P_ROPE ? 8 : 1];
            if constexpr (EPI == EPI_P_ROPE) {
                int mt, nt;
                order.at(t, mt, nt);
                rope_table_rows(p, mt * 256 + (int)rank * 128 + q * 32 + lane, nt * BN + half * 64, tab);
            }
            const bool ok = tc::mbar_wait_until(&acc_full[buf], (uint32_t)((i >> 1) & 1), deadline, abort_flag);
            if (!__all_sync(0xffffffffu, ok)) {
                if (!*abort_flag) atomicCAS(&g_gemm_status, 0, ERR_EPILOGUE | (blockIdx.x << 8));
                *abort_flag = 1;
                if constexpr (SPLIT)
                    for (; t < total; t += npairs)
                        if (lane == 0) split_k_arrive(p, t, S, (int)rank * 8 + (warp - 2));
                break;
            }
            tc::tc_fence_after_sync();
            int mt, nt;
            order.at(SPLIT ? t / S : t, mt, nt);
            const uint32_t t_acc = tmem + buf * Cfg::ACC_STRIDE + lane_off;
            bool finish = true;
            if constexpr (SPLIT)
                finish = split_k_sum<BN / 2>(p, t_acc + half * (BN / 2), t, S, (int)rank * 8 + (warp - 2));
            const int m_base = mt * 256 + (int)rank * 128 + q * 32;
            if constexpr (Cfg::OVERLAP) {
                // shared with the other accumulator: the last 64 columns of the first, the first 64 of the second.  Their warps
                // arrive when they have read them, the others now: they are through with the tiles before this one
                const bool shared = half != buf;
                const uint32_t bar = tc::dsmem_map(tc::smem_u32(&acc_empty[buf]), 0);
                if (!shared) {
                    tc::tc_fence_before_sync();
                    tc::mbar_arrive_cluster(bar);
                }
                const int flip = buf == 0 && half == 1 ? 64 : 0;
                const int c0 = half * 128 + flip, c1 = half * 128 + (64 - flip);
                epilogue_rows<EPI, 64>(p, t_acc + c0, m_base, nt * BN + c0, stg, lines, alpha, inv_os, shared ? bar : 0u);
                epilogue_rows<EPI, 64>(p, t_acc + c1, m_base, nt * BN + c1, stg, lines, alpha, inv_os);
                continue;
            } else if constexpr (EPI == EPI_P_ROPE)
                epilogue_rope_rows(p, t_acc + half * 64, m_base + lane, nt * BN + half * 64, alpha, pos, tab);
            else if constexpr (EPI == EPI_P_GEGLU_FP8)
                epilogue_geglu_rows(p, t_acc + half * 32, t_acc + BN / 2 + half * 32, m_base, nt * (BN / 2) + half * 32, alpha,
                                    inv_os);
            else if constexpr (BN == 192) {                  // whole 64-column blocks: 128 + 64
                if (half == 0) epilogue_rows<EPI, 128>(p, t_acc, m_base, nt * BN, stg, lines, alpha, inv_os);
                else epilogue_rows<EPI, 64>(p, t_acc + 128, m_base, nt * BN + 128, stg, lines, alpha, inv_os);
            } else if (finish)
                epilogue_rows<EPI, BN / 2>(p, t_acc + half * (BN / 2), m_base, nt * BN + half * (BN / 2), stg, lines, alpha,
                                           inv_os);
            tc::tc_fence_before_sync();
            tc::mbar_arrive_cluster(tc::dsmem_map(tc::smem_u32(&acc_empty[buf]), 0));
        }
    }
    __syncwarp();
    tc::tc_fence_before_sync();
    tc::cluster_sync_all();                    // the leader's MMAs read the peer's shared memory until the end
    if (warp == 1) tc::tmem_dealloc_pair(tmem, Cfg::TMEM_COLS);
}

template <int BN, int EPI, bool SPLIT = false, bool FP4 = false>
static int launch_gemm_pair(const void* A, const void* W, GemmParams p, int K, cudaStream_t stream) {
    using Cfg = GemmPairCfg<BN, FP4>;
    static PerDeviceOnce attr_once;
    int attr_dev = 0;
    const int sms = device_sm_count();
    if (attr_once.need(attr_dev)) {
        cudaError_t e = cudaFuncSetAttribute(gemm_fp8_pair_kernel<BN, EPI, SPLIT, FP4>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
        if (e != cudaSuccess) return FRT_CUDA_ERR(e);
        attr_once.set(attr_dev);
    }
    CUtensorMap tmA, tmW;
    PairScaleMaps<FP4> sfm;
    const uint64_t row_bytes = FP4 ? (uint64_t)K / 2 : (uint64_t)K;
    int rc = get_tmap_2d_u8(&tmA, A, (uint64_t)p.M, row_bytes, row_bytes, 128);
    if (rc) return rc;
    rc = get_tmap_2d_u8(&tmW, W, (uint64_t)p.N, row_bytes, row_bytes, BN / 2);
    if (rc) return rc;
    if constexpr (FP4) {
        rc = get_tmap_sf(&sfm.a, p.sf_lane, (p.M + 127) / 128, K / 64, 1);
        if (rc) return rc;
        rc = get_tmap_sf(&sfm.w, p.sf_col, (p.N + 127) / 128, K / 64, Cfg::SFB_ROWS);
        if (rc) return rc;
    }
    const int m_tiles = (p.M + 255) / 256, n_tiles = (p.N + BN - 1) / BN, total = m_tiles * n_tiles;
    p.tile_gm = tile_group(m_tiles, n_tiles, 256, BN, sms / 2);
    const int units = SPLIT ? total * p.ksplits : total;
    const int pairs = units < sms / 2 ? units : sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(64 + pair_epi_threads<EPI>());
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 2;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;    // nothing global is read before the wait
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
    cfg.attrs = attr;
    cfg.numAttrs = na;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_fp8_pair_kernel<BN, EPI, SPLIT, FP4>, tmA, tmW, p, sfm);
    return e == cudaSuccess ? FRT_OK : FRT_CUDA_ERR(e);
}
