"""The fused finishes of the projections store 8 results at a time (16 bytes of bf16, 8 of FP8) and read the rotary table in pieces of
16 bytes.  Shapes and pointers that do not fit are refused on the host -- seen here with no rows, where nothing is launched."""
import pytest

from flashrt_b200 import _lib

A = 4096                                                   # stands for an aligned device pointer; never read


def _fp8(rope=A, q=A, k=A, v=A, dims=(64, 8, 8, 8)):
    return "frt_b200_gemm_fp8_nt_rope_split", (A, A, 0, 128, None, None, rope, q, k, v, None, *dims, 0, 0, None)


def _nvfp4(rope=A, q=A, k=A, v=A, dims=(64, 8, 8, 8)):
    return "frt_b200_gemm_nvfp4_nt_rope_split", (A, A, A, A, 0, 256, 1.0, rope, q, k, v, None, *dims, 0, 0, None)


def _batched(rope=A, q=A, k=A, v=A, dims=(64, 8, 8, 8)):
    return "frt_b200_gemm_fp8_nt_rope_split_batched", (A, A, 0, 128, None, None, None, 0, 1e-6, None, rope, q, k, v, None, *dims, 0, 0,
                                                       0, 0, None)


def _normed(rope=A, q=A, k=A, v=A, dims=(64, 8, 8, 8)):
    return "frt_b200_norm_gemm_fp8_nt_rope_split", (A, A, 1, A, 1e-6, A, 0, 128, A, None, rope, q, k, v, None, *dims, 0, 0, None)


@pytest.mark.parametrize("call", [_fp8, _nvfp4, _batched, _normed])
def test_rope_finish(call):
    status = lambda **kw: _lib.call_status(call(**kw)[0], *call(**kw)[1])  # noqa: E731
    assert status() == 0
    assert status(dims=(64, 16, 8, 16)) == 0
    for dims in ((8, 4, 4, 4), (64, 8, 4, 8), (24, 12, 12, 12), (2, 2, 2, 2)):        # head dim or V width no multiple of 8
        assert status(dims=dims) == -2, dims
    for name in ("rope", "q", "k", "v"):
        for off in (2, 8):
            assert status(**{name: A + off}) == -1, (name, off)


@pytest.mark.parametrize("name,args", [
    ("frt_b200_gemm_fp8_nt_geglu_fp8", lambda out: (A, A, out, 0, 128, 128, None, None, A, 0, 0, None)),
    ("frt_b200_gemm_fp8_nt_geglu_fp8_rowscale", lambda out: (A, A, out, 0, 128, 128, None, None, A, 1, 1e-6, A, A, 0, 0, None)),
    ("frt_b200_norm_gemm_fp8_nt_geglu_fp8", lambda out: (A, A, 1, A, 1e-6, A, out, 0, 128, 128, A, None, A, 0, 0, None))])
def test_geglu_finish(name, args):
    assert _lib.call_status(name, *args(A + 8)) == 0
    for off in (1, 4):
        assert _lib.call_status(name, *args(A + off)) == -1
