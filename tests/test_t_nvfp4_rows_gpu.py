"""NVFP4 products of 65 to 256 rows with weights fetched early: a last tile of one row, of weight rows that end inside a tile, short
and long K.  The quantiser of few rows.  (The form of such products for chains of launches: test_u_nvfp4_chain_flag_gpu.py.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from test_h_nvfp4_gpu import _check, _operand  # noqa: E402


@pytest.mark.parametrize("M", [65, 100, 128, 129, 193, 256])
@pytest.mark.parametrize("N,K", [(1024, 2048), (1024, 4096), (72, 256), (1000, 1792), (2560, 1024), (1024, 14336)])
def test_rows_in_a_chain(M, N, K):
    from flashrt_b200 import _lib, flash_rt_kernels as fvk
    from gpu_util import Dev, zeros
    rng = np.random.default_rng(M + N + K)
    Ap, Asf = _operand(rng, M, K, 1.0)
    Wp, Wsf = _operand(rng, N, K, 0.02)
    bias = O.f32_to_bf16_bits((rng.standard_normal(N) * 0.1).astype(np.float32))
    d, d_b, d_o = [Dev(Ap), Dev(Asf), Dev(Wp), Dev(Wsf)], Dev(bias), zeros((M, N), np.uint16)
    _lib.call("frt_b200_gemm_nvfp4_nt", d[0].ptr, d[1].ptr, d[2].ptr, d[3].ptr, d_o.ptr, M, N, K, 1.0, None, d_b.ptr, 0, 1, 0)
    assert fvk.tensor_core_status() == 0
    _check(d_o.get(), O.gemm_nvfp4(Ap, Asf, Wp, Wsf, bias=bias, want_f32=True))


@pytest.mark.parametrize("rows,D", [(1, 16), (3, 48), (50, 2048), (200, 2048), (257, 4096), (300, 4096)])
@pytest.mark.parametrize("global_scale", [None, 0.37])
def test_quantiser_on_four_lanes(rows, D, global_scale):
    """Both sides of the line between the two forms, partial blocks of threads, with and without the global scale."""
    from flashrt_b200 import _lib
    from gpu_util import Dev, f32, zeros
    rng = np.random.default_rng(rows + D)
    x = O.f32_to_bf16_bits(rng.standard_normal((rows, D)).astype(np.float32))
    ref_p, ref_sf = O.quantize_nvfp4(x, 1, **({} if global_scale is None else dict(global_scale=global_scale)))
    d_x, d_p, d_sf = Dev(x), zeros(ref_p.shape, np.uint8), zeros(ref_sf.shape, np.uint8)
    g = None if global_scale is None else f32(global_scale)
    _lib.call("frt_b200_quantize_nvfp4", d_x.ptr, d_p.ptr, d_sf.ptr, rows, D, 1, g.ptr if g else None, 0, 0)
    assert np.array_equal(d_p.get(), ref_p) and np.array_equal(d_sf.get(), ref_sf)
