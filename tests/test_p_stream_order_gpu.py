"""Inputs that the caller's stream has not finished writing when a call is made: the model's own stream has to wait for them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


def _late(value):
    """A tensor that becomes ``value`` on the current stream some 50 ms after this returns, and is zero until then."""
    t = torch.zeros_like(value)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)
    t.copy_(value)
    return t


def test_expert_calibration_waits_for_its_samples():
    from flashrt_b200 import load_model
    from flashrt_b200.pi05_decoder import synthetic_state_dict
    model = load_model(synthetic_state_dict(seed=0, layers=2), config="pi05", layers=2, chunk_size=16, prefix_len=64)
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s, dtype=torch.float32: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    k, v, noise = r(2, 64, 256, dtype=BF16), r(2, 64, 256, dtype=BF16), r(16, 32)
    p = model._fe.pipeline
    model.set_prefix(k, v)
    torch.cuda.synchronize()
    model.calibrate([noise])
    want = [t.clone() for t in p.scale_tables()]
    model.calibrate([_late(noise)])
    for a, b in zip(p.scale_tables(), want):
        assert torch.equal(a, b)


def test_encoder_calibration_waits_for_its_samples():
    from flashrt_b200.pi05_prefix import Pi05PrefixEncoderB200
    enc = Pi05PrefixEncoderB200("synthetic:0", layers=2, max_seq=64)
    embeds = torch.randn(64, 2048, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(BF16)
    torch.cuda.synchronize()
    enc.calibrate([embeds])
    want = enc.act_scale.clone()
    enc.calibrate([_late(embeds)])
    assert torch.equal(enc.act_scale, want)


@pytest.mark.parametrize("precision", ["fp8", "nvfp4"])
def test_models_start_behind_the_stream_that_loaded_them(precision, monkeypatch):
    """Weights, tables and buffers are written on the caller's stream; the model's own stream waits for them, whatever call
    comes first."""
    from flashrt_b200 import load_model
    from flashrt_b200.pi05_decoder import synthetic_state_dict
    from flashrt_b200.pi05_prefix import Pi05PrefixEncoderB200
    waits, wait = [], torch.cuda.Stream.wait_stream
    monkeypatch.setattr(torch.cuda.Stream, "wait_stream", lambda s, other: (waits.append((s, other)), wait(s, other))[1])
    with torch.cuda.stream(torch.cuda.Stream()):
        here = torch.cuda.current_stream()
        fe = load_model(synthetic_state_dict(seed=0, layers=1), config="pi05", layers=1, chunk_size=16, prefix_len=64,
                        precision=precision)._fe
        enc = Pi05PrefixEncoderB200("synthetic:0", layers=1, max_seq=64)
    assert (fe.stream, here) in waits and (enc.stream, here) in waits
