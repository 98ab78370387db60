"""Both sides of the lines between forms of one kernel: the quantiser on four lanes a block and on one thread, the gated-residual
finish in items of four features and of eight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from test_h_nvfp4_gpu import _edge_rows  # noqa: E402
from test_m_gemm_tok_gpu import _fp8_operand  # noqa: E402


@pytest.mark.parametrize("family", [0, 1])
@pytest.mark.parametrize("global_scale", [None, 0.0371])
@pytest.mark.parametrize("D,over", [(4096, 0), (4096, 1), (1040, 1), (16, 0)])
def test_quantiser_around_the_line(family, global_scale, D, over):
    """The most rows that four lanes a block take (2048 threads an SM), and some more: ties, zero, tiny and huge blocks."""
    import torch
    from flashrt_b200 import _lib
    from gpu_util import Dev, f32, zeros
    rows = torch.cuda.get_device_properties(0).multi_processor_count * 2048 // (D // 4) + 5 * over
    x = _edge_rows(np.random.default_rng(D + family), rows, D)
    ref_p, ref_sf = O.quantize_nvfp4(x, family, **({} if global_scale is None else dict(global_scale=global_scale)))
    d_x, d_p, d_sf = Dev(x), zeros(ref_p.shape, np.uint8), zeros(ref_sf.shape, np.uint8)
    g = None if global_scale is None else f32(global_scale)
    _lib.call("frt_b200_quantize_nvfp4", d_x.ptr, d_p.ptr, d_sf.ptr, rows, D, family, g.ptr if g else None, 0, 0)
    assert np.array_equal(d_sf.get(), ref_sf)
    assert np.array_equal(d_p.get(), ref_p)


@pytest.mark.parametrize("splits,per", [(8, 9), (8, 16), (4, 9), (4, 16), (4, 17), (2, 9), (2, 17), (1, 9)])
@pytest.mark.parametrize("short", [0, 3])
def test_narrow_residual_finish_gives_the_bits_of_the_wide_one(splits, per, short):
    """At most eight tokens a rank: items of four features.  The same rows among more (the same K split) take items of eight: residual,
    next operand and row statistics byte for byte."""
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import Dev, f32, rand_bf16, zeros
    rng = np.random.default_rng(splits * 100 + per)
    few, M, N, K = 8 * splits - min(short, 8 * splits - 1), per * splits, 1024, 2048
    A, sa = _fp8_operand(rng, M, K, 1.0)
    W, sb = _fp8_operand(rng, N, K, 0.02)
    res0, gate, mod = rand_bf16(rng, (M, N), 1.0), rand_bf16(rng, (N,), 0.5), rand_bf16(rng, (N,), 0.3)
    d_W, d_sa, d_sb, d_gate, d_mod, d_q8s = Dev(W), f32(sa), f32(sb), Dev(gate), Dev(mod), f32(0.013)
    g, got = fvk.GemmRunner(), []
    for rows in (few, M):
        d_A, d_res, d_stats, d_q8 = Dev(A[:rows]), Dev(res0[:rows]), zeros((16, 128), np.float32), zeros((rows, N), np.uint8)
        n = g.fp8_nt_dev_gate_residual(d_A.ptr, d_W.ptr, rows, N, K, d_sa.ptr, d_sb.ptr, d_res.ptr, d_gate.ptr, d_stats.ptr, 0,
                                       splits=splits, tile_n=64, next_scale=d_mod.ptr, q8_out=d_q8.ptr, d_scale_q8=d_q8s.ptr)
        assert n == 16
        got.append((d_res.get()[:few], d_q8.get()[:few], d_stats.get()[:, :few].view(np.uint32)))
    assert fvk.tensor_core_status() == 0
    assert (got[0][2] != 0).all()
    for narrow, wide in zip(*got):
        assert np.array_equal(narrow, wide)
