"""NVFP4 products of 65 to 256 rows: early reads (flag bit 0) change no bits, the fused QKV product gives the bytes of the plain
one with and without them, and the form for chains of launches (flag bit 2) is right on its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from test_h_nvfp4_gpu import _check, _operand  # noqa: E402


def _order_operands(rng, M, N, K):
    """Operands whose sums depend on their order: the first block of 16 and the one in the middle of K are 64 times the rest and
    cancel each other, so small terms are rounded at the size of the large partial sum where both lie in one chain of sums
    and not where they lie in two."""
    a, w = (rng.standard_normal((r, K)).astype(np.float32) for r in (M, N))
    mid = K // 2
    a[:, :16] = 64.0 * rng.standard_normal((M, 16)).astype(np.float32)
    w[:, :16] = 64.0 * rng.standard_normal((N, 16)).astype(np.float32)
    a[:, mid:mid + 16], w[:, mid:mid + 16] = a[:, :16], -w[:, :16]
    (ap, asf), (wp, wsf) = (O.quantize_nvfp4(O.f32_to_bf16_bits(x), 1) for x in (a, w))
    return ap, asf, wp, wsf


def _product(d, M, N, K, splits, flags, bias=None, d_alpha=None, alpha=1.0, offset=0):
    """The product into a buffer that starts `offset` elements behind an aligned address."""
    from flashrt_b200 import _lib, flash_rt_kernels as fvk
    from gpu_util import zeros
    out = zeros((M * N + offset,), np.uint16)
    _lib.call("frt_b200_gemm_nvfp4_nt", *(x.ptr for x in d), out.ptr + 2 * offset, M, N, K, alpha, d_alpha, bias, splits, flags, 0)
    assert fvk.tensor_core_status() == 0
    return out.get()[offset:].reshape(M, N)


@pytest.mark.parametrize("M", [65, 100, 129, 200, 256])
@pytest.mark.parametrize("N,K", [(640, 1024), (1024, 2048), (1024, 4096), (2560, 1024)])
def test_early_reads_change_no_bits(M, N, K):
    from gpu_util import Dev
    d = [Dev(x) for x in _order_operands(np.random.default_rng(M + N + K), M, N, K)]
    assert np.array_equal(_product(d, M, N, K, 0, 0), _product(d, M, N, K, 0, 1))


@pytest.mark.parametrize("M,k_dim", [(65, 64), (100, 128), (128, 64), (200, 256), (256, 64)])
@pytest.mark.parametrize("pdl", [False, True])
def test_fused_qkv_equals_the_pair_of_launches(M, k_dim, pdl):
    from flashrt_b200 import flash_rt_fp4 as fp4, flash_rt_kernels as fvk
    from gpu_util import Dev, rand_bf16, zeros
    rng = np.random.default_rng(M + k_dim)
    K, q_dim, hd, pos = 1024, 8 * k_dim, k_dim, 5
    N = q_dim + 2 * k_dim
    d = [Dev(x) for x in _order_operands(rng, M, N, K)]
    d_rope, d_pos, d_qkv = Dev(rand_bf16(rng, (M, hd), 0.7)), Dev(np.array([pos], np.int32)), zeros((M, N), np.uint16)
    out = [[zeros((M, q_dim), np.uint16), zeros((pos + M, k_dim), np.uint16), zeros((pos + M, k_dim), np.uint16)]
           for _ in range(2)]
    assert fp4.cutlass_fp4_gemm_variant(0, *(x.ptr for x in d), d_qkv.ptr, M, N, K, 0.5, pdl=pdl) == 0
    fvk.qkv_split_rope(d_qkv.ptr, d_rope.ptr, out[0][0].ptr, out[0][1].ptr + pos * k_dim * 2,
                       out[0][2].ptr + pos * k_dim * 2, M, q_dim, k_dim, k_dim, hd, 0)
    assert fp4.cutlass_fp4_gemm_rope_split(*(x.ptr for x in d), d_rope.ptr, *(x.ptr for x in out[1]), M, K, q_dim, k_dim,
                                           k_dim, hd, devpos=d_pos.ptr, alpha=0.5, pdl=pdl) == 0
    assert fvk.tensor_core_status() == 0
    for a, b in zip(*out):
        assert np.array_equal(a.get(), b.get())


def _exact_operand(rng, rows, K):
    """Elements of the e2m1 set with a power-of-two scale per (64 rows, block): every product and every sum of them is exact."""
    x = rng.choice(np.array([-4, -3, -2, -1, 0, 1, 2, 3, 4, 6, -6], np.float32), (rows, K))
    x[:, ::16] = 6.0                                       # the largest of the block: its scale is the power of two
    e = rng.integers(-2, 3, ((rows + 63) // 64, K // 16))
    e[:, 0] += np.arange(e.shape[0]) % 2                   # neighbouring groups of 64 rows never agree
    return O.quantize_nvfp4((x * np.repeat(np.repeat(np.exp2(e), 16, axis=1), 64, axis=0)[:rows]).astype(np.float32), 1)


CHAIN = [(65, 1024, 2048), (100, 1024, 4096), (128, 72, 256), (129, 1024, 2048), (193, 1000, 1792), (256, 1024, 4096),
         (200, 520, 512), (100, 2560, 1024)]


@pytest.mark.parametrize("M,N,K", CHAIN)
@pytest.mark.parametrize("pdl", [0, 1])
def test_chain_form_is_exact_on_exact_products(M, N, K, pdl):
    """m-tiles of 64 rows, odd ones on the upper half of the operand and of the scale atoms, a last tile of one row: bit for bit."""
    from gpu_util import Dev
    rng = np.random.default_rng(M + N + K)
    (ap, asf), (wp, wsf) = _exact_operand(rng, M, K), _exact_operand(rng, N, K)
    d = [Dev(x) for x in (ap, asf, wp, wsf)]
    assert np.array_equal(_product(d, M, N, K, 0, 4 | pdl, alpha=0.125), O.gemm_nvfp4(ap, asf, wp, wsf, alpha=0.125))


@pytest.mark.parametrize("M,N,K", CHAIN)
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_chain_form_with_device_alpha_bias_and_any_alignment(M, N, K, offset):
    """A device scalar, a bias and a result that starts 2 or 8 bytes behind a 16-byte boundary: what stands beside it stays."""
    from flashrt_b200 import _lib, flash_rt_kernels as fvk
    from gpu_util import Dev, f32, zeros
    rng = np.random.default_rng(M + N + K + offset)
    (ap, asf), (wp, wsf) = _operand(rng, M, K, 1.0), _operand(rng, N, K, 0.02)
    bias = O.f32_to_bf16_bits((rng.standard_normal(N + 1) * 0.1).astype(np.float32))
    d, d_b, g = [Dev(x) for x in (ap, asf, wp, wsf)], Dev(bias), f32(0.5)
    out = Dev(np.full((M * N + offset + 8,), 0x7fc1, np.uint16))
    _lib.call("frt_b200_gemm_nvfp4_nt", *(x.ptr for x in d), out.ptr + 2 * offset, M, N, K, 2.0, g.ptr, d_b.ptr + 2 * (offset & 1),
              0, 5, 0)
    assert fvk.tensor_core_status() == 0
    got = out.get()
    _check(got[offset:offset + M * N].reshape(M, N),
           O.gemm_nvfp4(ap, asf, wp, wsf, bias=bias[offset & 1:][:N], want_f32=True))
    assert (got[:offset] == 0x7fc1).all() and (got[offset + M * N:] == 0x7fc1).all()


@pytest.mark.parametrize("M,N,K,chain", [(100, 1024, 2048, True), (256, 1024, 4096, True), (65, 640, 1024, True),
                                         (64, 1024, 2048, False), (257, 1024, 2048, False), (100, 8192, 1024, False),
                                         (100, 1020, 2048, False)])
def test_where_the_chain_form_runs(M, N, K, chain):
    """Its K splits show in the order of the sums; outside its range the flag changes nothing."""
    from gpu_util import Dev
    d = [Dev(x) for x in _order_operands(np.random.default_rng(M + N + K), M, N, K)]
    assert np.array_equal(_product(d, M, N, K, 0, 1), _product(d, M, N, K, 0, 5)) != chain
    for other in (2, 0x100):                               # a kernel that is asked for stays the one that runs
        assert np.array_equal(_product(d, M, N, K, 0, 1 | other), _product(d, M, N, K, 0, 5 | other))
    assert np.array_equal(_product(d, M, N, K, 1, 1), _product(d, M, N, K, 1, 5))


@pytest.mark.parametrize("M,N,K", [(65, 4736, 2048), (65, 4736, 1024), (80, 3584, 1024), (192, 2560, 2048), (65, 2560, 2048),
                                   (128, 4736, 2048), (192, 2560, 1280)])
def test_chain_form_stays_off_where_pairs_are_faster(M, N, K):
    """Unsplit products of many CTAs.  The unsplit form on the token-major kernel and the pairs add in the same order, so the
    kernel is read from the launch."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    from gpu_util import Dev
    d = [Dev(x) for x in _order_operands(np.random.default_rng(1), M, N, K)]
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        _product(d, M, N, K, 0, 5)
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages() if "gemm" in e.key]
    assert names and all("pair" in n for n in names), names
