"""What the header says of fused launches against the launches they replace, at row counts whose unhinted product leaves the
split-K kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_b_gemm_gpu import _fp8_operand  # noqa: E402


@pytest.mark.parametrize("M,splits", [(17, 1), (50, 8), (100, 4), (130, 2), (200, 4), (256, 1)])
def test_fused_projections_equal_two_launches_at_a_given_split(M, splits):
    """The same `splits` in {1, 2, 4, 8}: QKV + RoPE, gate|up + GeGLU, and the (K, N) weight layout give the bytes of the
    plain product and the launch behind it."""
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, f32, rand_bf16, zeros
    rng = np.random.default_rng(M + splits)
    K, q_dim, k_dim, hd, half = 1024, 1536, 256, 256, 1024
    N = q_dim + 2 * k_dim
    A, sa = _fp8_operand(rng, M, K, 1.0)
    W, sb = _fp8_operand(rng, N, K, 0.03)
    rope = rand_bf16(rng, (M, hd))
    d_A, d_W, d_Wt, d_sa, d_sb, d_so, d_rope = (Dev(A), Dev(W), Dev(np.ascontiguousarray(W.T)), f32(sa), f32(sb), f32(0.004),
                                                Dev(rope))
    g = fvk.GemmRunner()
    plain, kn = zeros((M, N), np.uint16), zeros((M, N), np.uint16)
    two = [zeros((M, d), np.uint16) for d in (q_dim, k_dim, k_dim)] + [zeros((M, half), np.uint8)]
    one = [zeros((M, d), np.uint16) for d in (q_dim, k_dim, k_dim)] + [zeros((M, half), np.uint8)]
    g.fp8_nt_dev(d_A.ptr, d_W.ptr, plain.ptr, M, N, K, d_sa.ptr, d_sb.ptr, 0, splits=splits)
    g.fp8_nn_dev(d_A.ptr, d_Wt.ptr, kn.ptr, M, N, K, d_sa.ptr, d_sb.ptr, 0, splits=splits)
    fvk.qkv_split_rope(plain.ptr, d_rope.ptr, two[0].ptr, two[1].ptr, two[2].ptr, M, q_dim, k_dim, k_dim, hd, 0)
    fvk.gate_geglu_merged_fp8(plain.ptr, two[3].ptr, M, half, d_so.ptr, 0)
    g.fp8_nt_dev_rope_split(d_A.ptr, d_W.ptr, M, K, d_sa.ptr, d_sb.ptr, d_rope.ptr, one[0].ptr, one[1].ptr, one[2].ptr, q_dim,
                            k_dim, k_dim, hd, 0, splits=splits)
    g.fp8_nt_dev_geglu_fp8(d_A.ptr, d_W.ptr, one[3].ptr, M, half, K, d_sa.ptr, d_sb.ptr, d_so.ptr, 0, splits=splits)
    assert fvk.tensor_core_status() == 0
    assert np.array_equal(plain.get(), kn.get()) and (two[3].get() != 0).mean() > 0.5
    for a, b in zip(two, one):
        assert np.array_equal(a.get(), b.get())
