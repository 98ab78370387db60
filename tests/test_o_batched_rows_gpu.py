"""GPU parity of the folded loop's launches at the row counts of a batch (65 .. 256 rows in one or more m-tiles), and of the
attention split chosen by size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from test_b_gemm_gpu import _check, _fp8_operand, _ref  # noqa: E402
from test_c_attention_gpu import _run  # noqa: E402


@pytest.mark.parametrize("batch,S,half", [(2, 33, True), (2, 64, True), (3, 43, False), (4, 64, False), (4, 50, True), (5, 13, False)])
def test_projections_of_a_batch(batch, S, half):
    """Row-scaled QKV (rope and cache rows per element), gated residual with the next operand and row-scaled gate|up at
    M = batch * S: the codes, statistics and residual of every row are those of its own element run alone."""
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, f32, rand_bf16, zeros
    rng = np.random.default_rng(batch * 100 + S)
    M, D, H, hd, rows = batch * S, 1024, 512, 256, S + 7
    q_dim, k_dim, v_dim = 512, 256, 256
    ld = 128 if M <= 128 else 256
    A, sa = _fp8_operand(rng, M, D, 1.0)
    Wq, sq = _fp8_operand(rng, q_dim + k_dim + v_dim, D, 0.02)
    Wg, sg = _fp8_operand(rng, 2 * H, D, 0.03)
    Wo, so = _fp8_operand(rng, D, D, 0.02)
    rope = rand_bf16(rng, (S, hd), 1.0)
    res0, gate, mod = rand_bf16(rng, (M, D), 1.0), rand_bf16(rng, (D,), 0.5), rand_bf16(rng, (D,), 0.3)
    ssq = (rng.random((16, M)) * D / 4.0).astype(np.float32)
    cq, cg = rng.standard_normal(q_dim + k_dim + v_dim).astype(np.float32), rng.standard_normal(2 * H).astype(np.float32)
    d_A, d_Wq, d_Wg, d_Wo, d_rope, d_gate, d_mod = (Dev(a) for a in (A, Wq, Wg, Wo, rope, gate, mod))
    d_sa, d_sq, d_sg, d_so, d_s8, d_cq, d_cg = f32(sa), f32(sq), f32(sg), f32(so), f32(0.013), Dev(cq), Dev(cg)
    g = fvk.GemmRunner()
    h = dict(half_tiles=half)

    def run(first, n):
        m = n * S
        pitch = 128 if m <= 128 else 256
        st = np.zeros((16, pitch), np.float32)
        st[:, :m] = ssq[:, first * S:first * S + m]
        d_st, d_a, d_res = Dev(st), Dev(A[first * S:first * S + m]), Dev(res0[first * S:first * S + m])
        Q, K, V = zeros((m, q_dim), np.uint16), zeros((n, rows, k_dim), np.uint16), zeros((n, rows, v_dim), np.uint16)
        hid, q8, so_ = zeros((m, H), np.uint8), zeros((m, D), np.uint8), Dev(np.full((16, pitch), -1.0, np.float32))
        g.fp8_nt_dev_rope_split_batched(d_a.ptr, d_Wq.ptr, m, D, d_sa.ptr, d_sq.ptr, d_st.ptr, 16, d_cq.ptr, d_rope.ptr,
                                        Q.ptr, K.ptr + 7 * k_dim * 2, V.ptr + 7 * v_dim * 2, q_dim, k_dim, v_dim, hd, S,
                                        rows * k_dim, 0, splits=2, tile_n=64, **h)
        g.fp8_nt_dev_geglu_fp8_rowscale(d_a.ptr, d_Wg.ptr, hid.ptr, m, H, D, d_sa.ptr, d_sg.ptr, d_st.ptr, 16, d_cg.ptr,
                                        d_s8.ptr, 0, splits=1, tile_n=128, **h)
        k = g.fp8_nt_dev_gate_residual(d_a.ptr, d_Wo.ptr, m, D, D, d_sa.ptr, d_so.ptr, d_res.ptr, d_gate.ptr, so_.ptr, 0,
                                       splits=4, tile_n=64, next_scale=d_mod.ptr, q8_out=q8.ptr, d_scale_q8=d_s8.ptr, **h)
        assert fvk.tensor_core_status() == 0 and k == 16
        return [a.get() for a in (Q, K, V, hid, q8, d_res)] + [so_.get()]

    whole = run(0, batch)
    assert (whole[6][:, M:] == -1.0).all() and whole[6].shape[1] == ld
    for e in range(batch):
        one = run(e, 1)
        for i in (0, 3, 4, 5):
            assert np.array_equal(whole[i][e * S:(e + 1) * S], one[i])
        assert np.array_equal(whole[1][e], one[1][0]) and np.array_equal(whole[2][e], one[2][0])
        assert np.array_equal(whole[6][:, e * S:(e + 1) * S], one[6][:, :S])
    rms = 1.0 / np.sqrt(ssq.astype(np.float64).sum(0) / D + 1e-6)
    v = (_ref(A, Wq, sa, sq).astype(np.float64) * rms[:, None] + cq[None, :])[:, q_dim + k_dim:]
    _check(whole[2][:, 7:].reshape(M, v_dim), v.astype(np.float32))


@pytest.mark.parametrize("B,Sq,Skv,extra", [(1, 20, 170, {}), (1, 60, 828, {}), (2, 50, 818, dict(fused_fp8=True)),
                                            (4, 50, 818, {}), (3, 24, 792, dict(seqused=70)), (1, 16, 64, {}),
                                            (4, 64, 150, {}), (1, 300, 300, {}), (1, 541, 541, dict(fused_fp8=True)),
                                            (1, 768, 768, {}), (1, 1040, 200, {})])
def test_attention_split_chosen_by_size(B, Sq, Skv, extra):
    """flags bit 4: a bound on the splits; whatever split and number of parts is chosen matches the oracle."""
    _run(B, Sq, Skv, 8, 1, 256, 8, seed=B + Sq, scratch=True, flags=16, **extra)


def test_fp8_batch4_agrees_with_single_runs():
    """200 rows per projection (two m-tiles, the rows of an element across them) through the whole captured loop."""
    import torch
    from flashrt_b200 import load_model
    from flashrt_b200.pi05_decoder import synthetic_state_dict
    from oracle import block_ref as R
    L = 2
    sd = synthetic_state_dict(seed=0, layers=L)
    k, v = (t.to(torch.bfloat16) for t in R.synthetic_prefix_kv(seed=1, layers=L, prefix_len=300))
    cal = [R.synthetic_noise(100 + j) for j in range(2)]
    noises = np.stack([R.synthetic_noise(10 + j).to(torch.bfloat16).float().numpy() for j in range(4)])
    models = []
    for b in (1, 4):
        m = load_model(sd, config="pi05", layers=L, num_steps=10, chunk_size=50, prefix_len=300, batch=b)
        m.set_prefix(k, v)
        m.calibrate([torch.stack([c] * b) if b > 1 else c for c in cal])
        models.append(m)
    got = models[1].predict(noise=noises)
    for j in range(4):
        one = models[0].predict(noise=noises[j])
        assert np.abs(got[j] - one).max() <= 3e-2 * float(np.sqrt((one ** 2).mean()))


@pytest.mark.parametrize("M,N,K", [(33, 256, 512), (65, 256, 512), (128, 384, 256), (200, 1024, 512), (256, 1024, 2560),
                                   (200, 6144, 256), (200, 16384, 256)])
def test_nvfp4_column_tiles(M, N, K):
    """Exact products with a different power-of-two scale in every block: column tiles of 64 (both halves of a 128-row group
    of scales), 128 and 256 tokens equal the oracle bit for bit."""
    from test_h_nvfp4_gpu import _run_gemm
    rng = np.random.default_rng(M + N)

    def make(rows):
        e = rng.integers(-3, 3, (rows, K // 16))
        x = rng.choice(np.array([-4, -3, -2, -1, 0, 1, 2, 3, 4, 6, -6], np.float32), (rows, K))
        x = x * np.repeat(np.exp2(e).astype(np.float32), 16, axis=1)
        x[:, ::16] = 6.0 * np.exp2(e).astype(np.float32)
        return O.quantize_nvfp4(x.astype(np.float32), 1)

    a, w = make(M), make(N)
    assert np.array_equal(_run_gemm(*a, *w, M, N, K, alpha=0.125), O.gemm_nvfp4(*a, *w, alpha=0.125))


@pytest.mark.parametrize("M,half,K", [(257, 128, 256), (300, 384, 1024), (768, 2048, 128), (2000, 1280, 512)])
def test_geglu_projection_of_many_rows(M, half, K):
    """M > 256: the pair kernel's GeGLU epilogue gives the bytes of product -> geglu_fp8, ragged rows included."""
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, f32, zeros
    rng = np.random.default_rng(M + half)
    A, sa = _fp8_operand(rng, M, K, 1.0)
    W, sb = _fp8_operand(rng, 2 * half, K, 0.05)
    d_A, d_W, d_sa, d_sb, d_so = Dev(A), Dev(W), f32(sa), f32(sb), f32(0.004)
    merged, two, one = zeros((M, 2 * half), np.uint16), zeros((M, half), np.uint8), Dev(np.full((M + 1, half), 0x5A, np.uint8))
    g = fvk.GemmRunner()
    g.fp8_nt_dev(d_A.ptr, d_W.ptr, merged.ptr, M, 2 * half, K, d_sa.ptr, d_sb.ptr)
    fvk.gate_geglu_merged_fp8(merged.ptr, two.ptr, M, half, d_so.ptr, 0)
    g.fp8_nt_dev_geglu_fp8(d_A.ptr, d_W.ptr, one.ptr, M, half, K, d_sa.ptr, d_sb.ptr, d_so.ptr)
    assert fvk.tensor_core_status() == 0
    assert np.array_equal(one.get()[:M], two.get()) and (one.get()[M] == 0x5A).all() and (two.get() != 0).mean() > 0.5


@pytest.mark.parametrize("used", [1, 65, 333, 818])
def test_attention_length_read_early(used):
    """kv_static_rows = -n: the splits share the chunks that hold keys; same bound against the oracle."""
    from flashrt_b200 import flash_rt_fa2 as fa2
    from gpu_util import Dev, rand_bf16, zeros
    rng = np.random.default_rng(used)
    S, T, H, D = 50, 818, 8, 256
    q, k, v = rand_bf16(rng, (1, S, H, D)), rand_bf16(rng, (1, T, 1, D)), rand_bf16(rng, (1, T, 1, D))
    d_q, d_k, d_v, d_o, d_u = Dev(q), Dev(k), Dev(v), zeros((1, S, H, D), np.uint16), Dev(np.array([used], np.int32))
    acc, lse, cnt = zeros((8, 1, H, S, D), np.float32), zeros((8, 1, H, S), np.float32), zeros((16,), np.int32)
    qs, ks = (S * H * D, H * D, D), (T * D, D, D)
    fa2.fwd_bf16_seqused_splitkv(d_q.ptr, d_k.ptr, d_v.ptr, d_o.ptr, 0, d_u.ptr, lse.ptr, acc.ptr, 1, S, T, H, 1, D, qs, ks,
                                 ks, qs, 1.0 / 16.0, 148, 0, kv_splits=8, counters=cnt.ptr, kv_static_rows=-S, pdl=True)
    ref, _ = O.attention(q, k, v, 1.0 / 16.0, used)
    got = O.bf16_bits_to_f32(d_o.get())
    assert fa2.attention_status() == 0
    assert (np.abs(got - ref) <= 2e-2 * np.sqrt((ref.astype(np.float64) ** 2).mean()) + np.abs(ref) * 2.0 ** -8).all()


@pytest.mark.parametrize("M,N,K,io,acc", [(50, 1024, 32, 1, False), (3, 30, 32, 0, True), (201, 1026, 32, 3, True),
                                          (50, 33, 32, 0, False), (5, 32, 1024, 2, True), (2, 40, 1500, 0, False)])
def test_action_projection_sums(M, N, K, io, acc):
    """Both forms of the small bf16 product: 16 interleaved K-slices added in order, then bias, then the old value."""
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, rand_bf16
    rng = np.random.default_rng(M + N + K)
    b, bias = rand_bf16(rng, (K, N), 0.5), rand_bf16(rng, (N,), 0.5)
    a = rng.standard_normal((M, K)).astype(np.float32) if io & 1 else rand_bf16(rng, (M, K))
    d = rng.standard_normal((M, N)).astype(np.float32) if io & 2 else rand_bf16(rng, (M, N))
    d_a, d_b, d_bias, d_d = Dev(a), Dev(b), Dev(bias), Dev(d)
    fvk.call("frt_b200_gemm_bf16_nn_small", d_a.ptr, d_b.ptr, d_d.ptr, d_bias.ptr, M, N, K, int(acc), io, 1, 0)
    af = O.bf16_bits_to_f32(O.f32_to_bf16_bits(a) if io & 1 else a)
    bf = O.bf16_bits_to_f32(b)
    s = np.zeros((M, N), np.float32)
    for q in range(16):
        part = np.zeros((M, N), np.float32)
        for k in range(q, K, 16):                       # products of two bf16 values are exact in fp64: one rounding per term
            part = (af[:, k:k + 1].astype(np.float64) * bf[k].astype(np.float64) + part).astype(np.float32)
        s = s + part
    s = s + O.bf16_bits_to_f32(bias)
    if acc:
        s = s + (d if io & 2 else O.bf16_bits_to_f32(d))
    got = d_d.get()
    assert np.array_equal(got, s if io & 2 else O.f32_to_bf16_bits(s))


@pytest.mark.parametrize("M,N,K", [(257, 256, 16384), (768, 2048, 16384), (541, 2000, 16400), (300, 2056, 12288), (768, 2048, 2048),
                                   (50, 1024, 4096)])
def test_split_k_product(M, N, K):
    """K split through a workspace: exact products (integers) give the oracle's bits, twice on the same counters."""
    import torch
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, f32, rand_bf16, zeros
    rng = np.random.default_rng(M + N + K)
    vals = np.array([-2, -1, 0, 1, 2], np.float32)
    e4 = lambda *s: torch.from_numpy(rng.choice(vals, s)).to(torch.float8_e4m3fn).view(torch.uint8).numpy()  # noqa: E731
    A, W, bias = e4(M, K), e4(N, K), rand_bf16(rng, (N,), 0.2)
    d_A, d_W, d_b, d_sa, d_sb = Dev(A), Dev(W), Dev(bias), f32(0.5), f32(0.25)
    ws, cnt = torch.empty(74 * 65536, dtype=torch.float32, device="cuda"), zeros((1184,), np.int32)
    plain = zeros((M, N), np.uint16)
    g = fvk.GemmRunner()
    g.fp8_nt_dev(d_A.ptr, d_W.ptr, plain.ptr, M, N, K, d_sa.ptr, d_sb.ptr, bias=d_b.ptr)
    _check(plain.get(), _ref(A, W, 0.5, 0.25, bias))
    for _ in range(2):
        d_D = Dev(np.full((M + 1, N), 0x5A5A, np.uint16))
        g.fp8_nt_dev_splitk(d_A.ptr, d_W.ptr, d_D.ptr, M, N, K, d_sa.ptr, d_sb.ptr, ws.data_ptr(), ws.numel() * 4, cnt.ptr,
                            bias=d_b.ptr)
        got = d_D.get()
        assert fvk.tensor_core_status() == 0
        assert np.array_equal(got[:M], plain.get()) and (got[M] == 0x5A5A).all() and (cnt.get() == 0).all()


@pytest.mark.parametrize("M,N,K", [(541, 9216, 2048), (2001, 3080, 2064), (1030, 2600, 2048)])
def test_pair_tiles_of_192_columns(M, N, K):
    """Sizes whose cheapest tile is 256 x 192, ragged in both directions: exact products plus bias give the oracle's bits."""
    import torch
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, f32, rand_bf16, zeros
    rng = np.random.default_rng(M + N)
    e4 = lambda *s: torch.from_numpy(rng.choice(np.array([-2, -1, 0, 1, 2], np.float32), s)).to(torch.float8_e4m3fn)  # noqa: E731
    A, W, bias = e4(M, K), e4(N, K), rand_bf16(rng, (N,), 0.5)
    d_A, d_W, d_b, d_sa, d_sb = Dev(A.view(torch.uint8).numpy()), Dev(W.view(torch.uint8).numpy()), Dev(bias), f32(0.5), f32(0.0625)
    d_D = Dev(np.full((M + 1, N), 0x5A5A, np.uint16))
    g = fvk.GemmRunner()
    g.fp8_nt_dev(d_A.ptr, d_W.ptr, d_D.ptr, M, N, K, d_sa.ptr, d_sb.ptr, bias=d_b.ptr)
    acc = (A.float().cuda() @ W.float().cuda().T).cpu().numpy() * np.float32(0.03125)          # integers: exact
    got = d_D.get()
    assert fvk.tensor_core_status() == 0 and (got[M] == 0x5A5A).all()
    assert np.array_equal(got[:M], O.f32_to_bf16_bits((acc + O.bf16_bits_to_f32(bias)).astype(np.float32)))
    # and bias + GELU + FP8 in the finish equals the separate launch
    d_mid, d_two, d_one, d_so = zeros((M, N), np.uint16), zeros((M, N), np.uint8), zeros((M, N), np.uint8), f32(0.05)
    g.fp8_nt_dev(d_A.ptr, d_W.ptr, d_mid.ptr, M, N, K, d_sa.ptr, d_sb.ptr)
    fvk.bias_gelu_quantize_fp8_static_bf16(d_mid.ptr, d_b.ptr, d_two.ptr, d_so.ptr, M, N, 0)
    g.fp8_nt_dev_bias_gelu_fp8(d_A.ptr, d_W.ptr, d_one.ptr, M, N, K, d_sa.ptr, d_sb.ptr, d_b.ptr, d_so.ptr, 0)
    assert np.array_equal(d_one.get(), d_two.get())
