"""Two-tile attention (head_dim 128) whose last wave goes as CTAs of one tile: against the fp64 oracle where all CTAs hold one tile, and,
with whole waves in front, against the same heads in calls of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_c_attention_gpu import _run  # noqa: E402


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv", [(1, 129, 128, 1, 1), (1, 257, 300, 3, 3), (2, 300, 129, 5, 5), (1, 70, 200, 8, 2)])
def test_one_tile_per_cta(B, Sq, Skv, Hq, Hkv):
    """An odd last tile, a CTA behind the last row, partial chunks, grouped heads."""
    _run(B, Sq, Skv, Hq, Hkv, 128, 1, seed=Sq + Skv)
    _run(B, Sq, Skv, Hq, Hkv, 128, 1, seed=Sq + Skv + 1, fused_fp8=True, seqused=Skv - 3)


def test_whole_waves_and_a_rest():
    from flashrt_b200 import flash_rt_fa2 as fa2
    from gpu_util import Dev, rand_bf16, zeros
    rng = np.random.default_rng(5)
    B, S, T, H, D = 1, 300, 200, 85, 128                       # 170 units of two tiles: one wave of 148 and 22 as 44 CTAs
    q, k, v = (rand_bf16(rng, (B, n, H, D)) for n in (S, T, T))
    d = [Dev(x) for x in (q, k, v)]
    o_all, o_each = zeros((B, S, H, D), np.uint16), zeros((B, S, H, D), np.uint16)
    qs, ks = (S * H * D, H * D, D), (T * H * D, H * D, D)
    for out, heads in ((o_all, [(0, H)]), (o_each, [(0, 74), (74, 11)])):      # 148 units; 22 units
        for h0, n in heads:
            off = 2 * h0 * D
            fa2.fwd_bf16(d[0].ptr + off, d[1].ptr + off, d[2].ptr + off, out.ptr + off, 0, 0, 0, B, S, T, n, n, D, qs, ks, ks, qs,
                         1.0 / np.sqrt(D), 148, 0, kv_splits=1)
    assert fa2.attention_status() == 0
    assert np.array_equal(o_all.get(), o_each.get())
