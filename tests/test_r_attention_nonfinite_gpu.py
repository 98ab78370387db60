"""Non-finite scores in the two-tile attention: keys at the places whose exponentials run on the fma pipe (pairs 3 and 7 of every
32 keys) and beside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402


def _attend(q, k, v, D):
    from flashrt_b200 import flash_rt_fa2 as fa2
    from gpu_util import Dev, zeros
    Sq, Skv = q.shape[1], k.shape[1]
    d_q, d_k, d_v = Dev(q), Dev(k), Dev(v)
    d_o, d_lse = zeros(q.shape, np.uint16), zeros((1, 1, Sq), np.float32)
    qs, ks = (Sq * D, D, D), (Skv * D, D, D)
    fa2.fwd_bf16(d_q.ptr, d_k.ptr, d_v.ptr, d_o.ptr, d_lse.ptr, 0, 0, 1, Sq, Skv, 1, 1, D, qs, ks, ks, qs, D ** -0.5, 148, 0,
                 kv_splits=1)
    got = d_o.get()
    assert fa2.attention_status() == 0
    return O.bf16_bits_to_f32(got)[0, :, 0], d_lse.get()[0, 0]


@pytest.mark.parametrize("key", [0, 6, 7, 15, 46, 133, 255])
def test_nan_and_infinite_scores(key):
    from gpu_util import rand_bf16
    rng = np.random.default_rng(key)
    D, Sq, Skv = 128, 300, 256
    q, k, v = (rand_bf16(rng, (1, n, 1, D)) for n in (Sq, Skv, Skv))
    bad = k.copy()
    bad[0, key, 0, 0] = 0x7FC0                                   # NaN in every row's score of this key
    out, lse = _attend(q, bad, v, D)
    assert np.isnan(out).all() and not np.isfinite(lse).any()
    bad[0, key, 0, 0] = 0x7F80                                   # +inf: score +-inf by the sign of the query's first element
    out, _ = _attend(q, bad, v, D)
    up = O.bf16_bits_to_f32(q)[0, :, 0, 0] > 0
    assert np.isnan(out[up]).all()
    keep = np.arange(Skv) != key                                 # -inf: the key has no weight
    ref, _ = O.attention(q, k[:, keep], v[:, keep], D ** -0.5, Skv - 1)
    ref = ref[0, :, 0]
    rms = np.sqrt((ref.astype(np.float64) ** 2).mean())
    # the bound of the finite cases: 2e-2 x RMS plus one bf16 ulp of the value (P and the result are stored in bf16)
    assert (np.abs(out[~up] - ref[~up]) <= 2e-2 * rms + np.abs(ref[~up]) * 2.0 ** -8).all()
