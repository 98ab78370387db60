"""The work whose time this repository answers for, as calls of its public entry points.

Kinds of case:
  act      one control step with a prefix from elsewhere: hand over the per-layer prefix keys / values of the new
           observation, run the ten-step denoise loop, get the actions on the host
  observe  the whole control step: prefix encoder on the observation's embeddings (into the loop's cache), then the loop
  video    one denoise step of the video DiT (two blocks of its stack: every block does the same work)
  linear   a normalised, quantised projection through the operator names: RMSNorm -> FP8 / NVFP4, then the GEMM

Weights, calibration and captured graphs belong to the loaded model, which a program keeps; they are the same for every
seed.  Observations, latents, noise and operator operands come from the seed.
"""
from __future__ import annotations

import functools
import math

import torch

from flashrt_b200 import flash_rt_fp4 as fp4
from flashrt_b200 import flash_rt_kernels as fvk
from flashrt_b200 import load_model
from flashrt_b200.pi05_decoder import synthetic_state_dict
from flashrt_b200.pi05_prefix import EP, Pi05PrefixEncoderB200
from flashrt_b200.wan_dit import WanDiTB200

DEV = "cuda:0"
BF16 = torch.bfloat16
LAYERS, STEPS = 18, 10           # depth of action expert and prefix encoder; Euler steps of the loop
D, H, QKV, QD, HD = 1024, 4096, 2560, 2048, 256              # action expert
ENC_D, ENC_H = 2048, 16384                                   # prefix encoder
WAN_D, WAN_F, WAN_T, WAN_TEXT, WAN_HEADS = 3072, 14336, 512, 4096, 24
WAN_BLOCKS = 2


def listed():
    return [
        # the robot's inner loop at batch 1: 50 actions against a 768-token prefix, FP8 (the default) and NVFP4
        {"name": "act_fp8", "kind": "act", "precision": "fp8", "batch": 1, "guided": False, "chunk": 50, "prefix": 768},
        {"name": "act_nvfp4", "kind": "act", "precision": "nvfp4", "batch": 1, "guided": False, "chunk": 50, "prefix": 768},
        # classifier-free guidance: a conditioned and an unconditioned prefix in one pass
        {"name": "act_fp8_guided", "kind": "act", "precision": "fp8", "batch": 2, "guided": True, "chunk": 50, "prefix": 768},
        # four robots served by one model
        {"name": "act_nvfp4_batch4", "kind": "act", "precision": "nvfp4", "batch": 4, "guided": False, "chunk": 50,
         "prefix": 768},
        # the whole control step: three camera images' worth of tokens, and a shorter odd prompt through the graph that
        # serves every length
        {"name": "observe_768", "kind": "observe", "chunk": 50, "prefix": 768, "room": 768, "fixed": False},
        {"name": "observe_541_of_768", "kind": "observe", "chunk": 50, "prefix": 541, "room": 768, "fixed": True},
        # the video DiT: full-length clip with its guidance pair (the largest work), and a short clip of odd size
        {"name": "video_13x30x52", "kind": "video", "batch": 2, "f": 13, "h": 30, "w": 52},
        {"name": "video_4x17x29", "kind": "video", "batch": 1, "f": 4, "h": 17, "w": 29},
        # operators: the smallest call (launches count), an ordinary one, a large one, and 4-bit operands at odd row count
        {"name": "linear_fp8_16", "kind": "linear", "format": "fp8", "m": 16, "n": 1024, "k": 1024},
        {"name": "linear_fp8_256", "kind": "linear", "format": "fp8", "m": 256, "n": 4096, "k": 1024},
        {"name": "linear_fp8_8192", "kind": "linear", "format": "fp8", "m": 8192, "n": 14336, "k": 3072},
        {"name": "linear_nvfp4_2501", "kind": "linear", "format": "nvfp4", "m": 2501, "n": 3072, "k": 3072},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["act", "act", "observe", "video", "linear", "linear"])
    if kind == "act":
        precision, batch = rng.choice(["fp8", "nvfp4"]), rng.choice([1, 1, 2, 3, 4])
        return {"kind": kind, "precision": precision, "batch": batch, "guided": batch == 2 and rng.random() < 0.5,
                "chunk": rng.randint(10, 64), "prefix": _log_int(rng, 96, 1024)}
    if kind == "observe":
        prefix, fixed = _log_int(rng, 96, 1024), rng.random() < 0.5
        return {"kind": kind, "chunk": rng.randint(10, 64), "prefix": prefix,
                "room": (768 if prefix <= 768 else 1024) if fixed else prefix, "fixed": fixed}
    if kind == "video":
        return {"kind": kind, "batch": rng.choice([1, 2]), "f": _log_int(rng, 1, 13), "h": rng.randint(12, 30),
                "w": rng.randint(12, 52)}
    return {"kind": kind, "format": rng.choice(["fp8", "nvfp4"]), "m": _log_int(rng, 8, 20480),
            "n": 16 * _log_int(rng, 64, 896), "k": 256 * _log_int(rng, 4, 56)}


# ------------------------------------------------------------------ what a program loads once
def _gpu_gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(gen, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=gen, device=DEV) * scale).to(dtype)


@functools.lru_cache(maxsize=1)
def _expert_weights():
    sd = synthetic_state_dict(0, LAYERS)
    return {k: v.to(DEV) if "_proj.weight" in k and "gemma_expert" in k else v for k, v in sd.items()}


@functools.lru_cache(maxsize=4)
def _expert(precision, batch, guided, chunk, prefix, fixed):
    model = load_model(_expert_weights(), config="pi05", precision=precision, batch=batch,
                       cfg_beta=1.5 if guided else None, chunk_size=chunk, prefix_len=prefix, fixed_shape=fixed)
    g = _gpu_gen(1)
    model.set_prefix(_randn(g, LAYERS, prefix, HD, dtype=BF16), _randn(g, LAYERS, prefix, HD, dtype=BF16))
    rows = chunk if guided else batch * chunk
    model.calibrate([_randn(g, rows, 32) for _ in range(2)])
    return model


@functools.lru_cache(maxsize=1)
def _encoder():
    g, sd = _gpu_gen(2), {}
    for i in range(LAYERS):
        p = EP.format(i=i)
        for name, rows, cols in (("self_attn.q_proj", QD, ENC_D), ("self_attn.k_proj", HD, ENC_D),
                                 ("self_attn.v_proj", HD, ENC_D), ("self_attn.o_proj", ENC_D, QD),
                                 ("mlp.gate_proj", ENC_H, ENC_D), ("mlp.up_proj", ENC_H, ENC_D),
                                 ("mlp.down_proj", ENC_D, ENC_H)):
            sd[f"{p}.{name}.weight"] = _randn(g, rows, cols, scale=0.02, dtype=BF16)
        for name in ("input_layernorm", "post_attention_layernorm"):
            sd[f"{p}.{name}.weight"] = _randn(g, ENC_D, scale=0.1)
    enc = Pi05PrefixEncoderB200(sd, layers=LAYERS, max_seq=1024)
    enc.calibrate([_randn(g, 1024, ENC_D, dtype=BF16) for _ in range(2)])
    return enc


@functools.lru_cache(maxsize=2)
def _video(batch, f, h, w):
    g = _gpu_gen(3)
    m = lambda *s: _randn(g, *s, scale=0.02)  # noqa: E731
    ones, blocks = torch.ones(WAN_D, device=DEV), []
    for _ in range(WAN_BLOCKS):
        b = {"modulation": m(6, WAN_D) * 5, "norm3_w": ones, "norm3_b": torch.zeros(WAN_D, device=DEV),
             "ck": m(WAN_D, WAN_TEXT), "cv": m(WAN_D, WAN_TEXT), "ffn1": m(WAN_F, WAN_D), "ffn2": m(WAN_D, WAN_F),
             "ffn1_b": m(WAN_F), "ffn2_b": m(WAN_D)}
        for n in ("q", "k", "v", "o", "cq", "co"):
            b[n] = m(WAN_D, WAN_D)
        for n in ("q_b", "k_b", "v_b", "o_b", "cq_b", "ck_b", "cv_b", "co_b"):
            b[n] = m(WAN_D)
        for n in ("norm_q", "norm_k", "norm_cq", "norm_ck"):
            b[n] = ones
        blocks.append(b)
    model = WanDiTB200({"blocks": blocks, "dim": WAN_D, "ffn": WAN_F, "text_dim": WAN_TEXT,
                        "head_dim": WAN_D // WAN_HEADS}, grid=(f, h, w), batch=batch, text_len=WAN_T)
    model.set_context(_randn(g, batch, WAN_T, WAN_TEXT))
    model.calibrate(_randn(g, batch, model.L, WAN_D, dtype=BF16), _randn(g, batch, 6, WAN_D, scale=0.3))
    return model


def _linear_weights(g, case):
    n, k = case["n"], case["k"]
    w = _randn(g, n, k, scale=0.02, dtype=BF16)
    if case["format"] == "fp8":
        sb = (w.abs().max().float() / 448.0).reshape(1)
        return {"w": (w.float() / sb).clamp(-448, 448).to(torch.float8_e4m3fn), "sb": sb}
    packed = torch.empty(n, k // 2, dtype=torch.uint8, device=DEV)
    sf = torch.zeros(fp4.sfa_size_bytes(n, k, True), dtype=torch.uint8, device=DEV)
    gs = (w.abs().max().float() / (448.0 * 6.0)).reshape(1)
    if fp4.quantize_fp4_dynamic_sfa_bf16_vec(w.data_ptr(), packed.data_ptr(), sf.data_ptr(), n, k, True,
                                             torch.cuda.current_stream().cuda_stream, d_global_scale=gs.data_ptr()):
        raise RuntimeError("weight quantisation failed")
    return {"w": packed, "sf": sf, "gs": gs, "alpha": float(gs)}


# ------------------------------------------------------------------ the contract
def prepare(case, seed):
    g, kind = _gpu_gen(1000 + seed), case["kind"]
    s = {"case": case}
    if kind == "act":
        b, p = case["batch"], case["prefix"]
        s["model"] = _expert(case["precision"], b, case["guided"], case["chunk"], p, False)
        s["k"], s["v"] = (_randn(g, LAYERS, b, p, HD, dtype=BF16) for _ in range(2))
        rows = (case["chunk"],) if b == 1 or case["guided"] else (b, case["chunk"])
        s["noise"] = _randn(g, *rows, 32).cpu().numpy()
    elif kind == "observe":
        s["encoder"] = _encoder()
        s["model"] = _expert("fp8", 1, False, case["chunk"], case["room"], case["fixed"])
        s["embeds"] = _randn(g, case["prefix"], ENC_D, dtype=BF16)
        s["noise"] = _randn(g, case["chunk"], 32).cpu().numpy()
    elif kind == "video":
        s["model"] = m = _video(case["batch"], case["f"], case["h"], case["w"])
        s["x"] = _randn(g, case["batch"], m.L, WAN_D, dtype=BF16)
        s["time"] = _randn(g, case["batch"], 6, WAN_D, scale=0.3)
    else:
        m, n, k = case["m"], case["n"], case["k"]
        x = _randn(g, m, k, dtype=BF16)
        s.update(_linear_weights(g, case), x=x, gamma=(1.0 + _randn(g, k, scale=0.1)).to(BF16), gemm=fvk.GemmRunner(),
                 out=torch.empty(m, n, dtype=BF16, device=DEV))
        if case["format"] == "fp8":
            xf = x.float()
            normed = xf * torch.rsqrt(xf.square().mean(-1, keepdim=True) + 1e-6) * s["gamma"].float()
            s["sa"] = (normed.abs().max() / 448.0).reshape(1)
            s["a"] = torch.empty(m, k, dtype=torch.uint8, device=DEV)
        else:
            s["a"] = torch.empty(m, k // 2, dtype=torch.uint8, device=DEV)
            s["a_sf"] = torch.zeros(fp4.sfa_size_bytes(m, k), dtype=torch.uint8, device=DEV)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "act":
        s["model"].set_prefix(s["k"], s["v"])
        return s["model"].predict(noise=s["noise"])
    if kind == "observe":
        s["model"].set_prefix_from_encoder(s["encoder"], s["embeds"])
        return s["model"].predict(noise=s["noise"])
    if kind == "video":
        return s["model"].step(s["x"], s["time"])
    m, n, k = case["m"], case["n"], case["k"]
    st = torch.cuda.current_stream().cuda_stream
    x, a, w, out = s["x"].data_ptr(), s["a"].data_ptr(), s["w"].data_ptr(), s["out"].data_ptr()
    if case["format"] == "fp8":
        sa = s["sa"].data_ptr()
        fvk.rms_norm_fp8(x, s["gamma"].data_ptr(), a, m, k, 1e-6, sa, st)
        s["gemm"].fp8_nt_dev(a, w, out, m, n, k, sa, s["sb"].data_ptr(), st)
    else:
        a_sf = s["a_sf"].data_ptr()
        fp4.rms_norm_fp4_sfa_bf16(x, a, a_sf, m, k, st, weight=s["gamma"].data_ptr())
        if fp4.cutlass_fp4_gemm_variant(0, a, a_sf, w, s["sf"].data_ptr(), out, m, n, k, s["alpha"], 0.0, st):
            raise RuntimeError("GEMM failed")
    return {"activations": s["a"], "out": s["out"]}


def work(case):
    kind = case["kind"]
    if kind in ("act", "observe"):
        nv, b = case.get("precision") == "nvfp4", case.get("batch", 1)
        m, keys = b * case["chunk"], case["prefix"] + case["chunk"]
        weights = D * (QKV + QD + 2 * H + H)
        # the steps depend on one another and the weights (311 MB in FP8) exceed what the chip holds: read every step
        nbytes = STEPS * LAYERS * (weights * (0.5625 if nv else 1.0) + b * 2 * keys * HD * 2)
        flops = STEPS * LAYERS * (2.0 * m * weights + 4.0 * m * keys * QD)
        if kind == "observe":
            p, attn_qkv = case["prefix"], ENC_D * QKV
            rest = ENC_D * (QD + 3 * ENC_H)
            nbytes += LAYERS * attn_qkv + (LAYERS - 1) * rest + p * (ENC_D * 2 + LAYERS * 2 * HD * 2)
            flops += 2.0 * p * (LAYERS * attn_qkv + (LAYERS - 1) * rest) + (LAYERS - 1) * 4.0 * p * p * QD
        return {"bytes": nbytes, "flops": flops}
    if kind == "video":
        tokens = case["f"] * case["h"] * case["w"]
        m = case["batch"] * tokens
        weights = WAN_D * (3 * WAN_D + 3 * WAN_D + 2 * WAN_F)
        kv_text = 2 * case["batch"] * WAN_T * WAN_D * 2
        return {"bytes": 2 * m * WAN_D * 2 + WAN_BLOCKS * (weights + kv_text),
                "flops": WAN_BLOCKS * (2.0 * m * weights + 4.0 * m * (tokens + WAN_T) * WAN_D)}
    m, n, k = case["m"], case["n"], case["k"]
    eb = 1.0 if case["format"] == "fp8" else 0.5625
    return {"bytes": m * k * 2 + eb * (m * k + n * k) + m * n * 2, "flops": 2.0 * m * n * k}


def tolerance(case):
    # A last-bit difference flips some codes of every quantiser behind it by a whole step (6 % in E4M3, up to 50 % in
    # e2m1), so two correct pipelines agree to a fraction of the formats' own error: the loops and the DiT repeat that
    # over tens of quantised projections.  A single projection of the same codes differs by its bf16 rounding only.
    if case["kind"] == "linear":
        return {"rel": 3e-3, "max": 1e-2}
    if case["kind"] == "video" or case.get("precision") == "nvfp4":
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 2e-2, "max": 0.3}
