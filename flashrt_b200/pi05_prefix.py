"""Prefix producer on B200: the Gemma-2B encoder layers that turn the prompt / image embeddings into the
per-layer prefix keys and values the action expert attends to.

Host-side mirror of the reference's ``Pi05Pipeline._encoder_layer`` / ``transformer_encoder``
(flash_rt/models/pi05/pipeline_rtx.py:1209-1435, fused-FP8 branch) and of the encoder part of the checkpoint
conversion (flash_rt/frontends/torch/pi05_rtx.py:178-214: q / k rows interleaved for adjacent-pair RoPE, the
``1 + w`` of both RMSNorms folded into the following projections in fp32).  It is the step in front of the denoise
path and reuses its kernels unchanged, at M = prefix length where the GEMMs turn compute-bound:

  B1  rms_norm_fp8 (first layer) / residual_add_rms_norm_fp8 -> QKV GEMM -> qkv_split_rope (K, V straight into the
      layer's cache rows; K carries its RoPE)
  B2  bidirectional attention over the prefix (8 query heads, one KV head, head_dim 256), FP8 copy fused
  B3  attention out-projection
  B4  residual_add_rms_norm_fp8 -> gate|up GEMM -> GeGLU -> FP8
  B5  down projection (its residual add is fused into the next layer's B1)
The last layer stops after B1: the encoder's product is the KV cache, not its hidden state.
The vision tower and the token embedding are outside this module: ``embeds`` (seq, 2048) is the input.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from . import flash_rt_fa2 as fa2
from . import flash_rt_kernels as fvk
from .weight_loader import (DictSource, FlatCat, FoldNorm, FusedGateUp, FusedQKV, Item, LayerBlock, ModelWeightSpec,
                            Quant, SafetensorsSource, WeightLoader)

ENC_D, ENC_H, ENC_NH, ENC_NKV, ENC_HD, ENC_L = 2048, 16384, 8, 1, 256, 18
QKV_N = (ENC_NH + 2 * ENC_NKV) * ENC_HD
BF16 = torch.bfloat16
ATTN_SPLITS = 4             # most key splits of the encoder's attention
SITES = ("qkv", "o", "gu", "d")
EP = "paligemma_with_expert.paligemma.model.language_model.layers.{i}"


def build_encoder_spec(layers: int = ENC_L) -> ModelWeightSpec:
    blk = LayerBlock(prefix_fmt="", num_layers=layers, name="encoder", items=[
        Item("qkv_w", FoldNorm(FusedQKV(q=f"{EP}.self_attn.q_proj.weight", k=f"{EP}.self_attn.k_proj.weight",
                                        v=f"{EP}.self_attn.v_proj.weight", interleave_q_heads=ENC_NH,
                                        interleave_k_heads=ENC_NKV), norm=f"{EP}.input_layernorm.weight"),
             [Quant()], FlatCat("w_qkv"), scale_into="ws_qkv"),
        Item("o_w", f"{EP}.self_attn.o_proj.weight", [Quant()], FlatCat("w_o"), scale_into="ws_o"),
        Item("gu_w", FoldNorm(FusedGateUp(gate=f"{EP}.mlp.gate_proj.weight", up=f"{EP}.mlp.up_proj.weight"),
                              norm=f"{EP}.post_attention_layernorm.weight"),
             [Quant()], FlatCat("w_gu"), scale_into="ws_gu"),
        Item("d_w", f"{EP}.mlp.down_proj.weight", [Quant()], FlatCat("w_d"), scale_into="ws_d"),
    ])
    return ModelWeightSpec(framework="torch", blocks=[blk], dims={"D": ENC_D, "H": ENC_H, "L": layers})


def synthetic_encoder_state_dict(seed: int = 0, layers: int = ENC_L) -> dict:
    """Random-init Gemma-2B encoder layers under the HF key names (matrices ~ N(0, 0.02), norm weights ~ N(0, 0.1))."""
    g = torch.Generator().manual_seed(seed)
    w = lambda *shape, s=0.02: torch.randn(*shape, generator=g) * s  # noqa: E731
    sd = {}
    for i in range(layers):
        p = EP.format(i=i)
        sd[f"{p}.self_attn.q_proj.weight"] = w(ENC_NH * ENC_HD, ENC_D)
        sd[f"{p}.self_attn.k_proj.weight"] = w(ENC_NKV * ENC_HD, ENC_D)
        sd[f"{p}.self_attn.v_proj.weight"] = w(ENC_NKV * ENC_HD, ENC_D)
        sd[f"{p}.self_attn.o_proj.weight"] = w(ENC_D, ENC_NH * ENC_HD)
        sd[f"{p}.mlp.gate_proj.weight"] = w(ENC_H, ENC_D)
        sd[f"{p}.mlp.up_proj.weight"] = w(ENC_H, ENC_D)
        sd[f"{p}.mlp.down_proj.weight"] = w(ENC_D, ENC_H)
        sd[f"{p}.input_layernorm.weight"] = w(ENC_D, s=0.1)
        sd[f"{p}.post_attention_layernorm.weight"] = w(ENC_D, s=0.1)
    return sd


def rope_rows(count: int) -> torch.Tensor:
    """bf16 (count, 256) rows [cos0, sin0, ...] for positions 0 .. count-1, theta 10000 (pipeline_rtx.py:473-505)."""
    inv_freq = 1.0 / (10000 ** (np.arange(0, ENC_HD, 2, dtype=np.float64) / ENC_HD))
    phase = np.arange(count, dtype=np.float64)[:, None] * inv_freq[None, :]
    tab = np.stack([np.cos(phase), np.sin(phase)], axis=-1).reshape(count, ENC_HD)
    return torch.from_numpy(tab.astype(np.float32)).to(BF16)


class Pi05PrefixEncoderB200:
    def __init__(self, checkpoint, *, layers: int = ENC_L, max_seq: int = 768, device: int = 0):
        if not torch.cuda.is_available():
            raise RuntimeError("flashrt_b200 needs a CUDA device (sm_100a); there is no CPU path")
        self.device = torch.device("cuda", device)
        torch.cuda.set_device(self.device)
        self.layers, self.max_seq = layers, max_seq
        if isinstance(checkpoint, dict):
            source = DictSource(checkpoint)
        elif isinstance(checkpoint, str) and checkpoint.startswith("synthetic"):
            seed = int(checkpoint.split(":")[1]) if ":" in checkpoint else 0
            source = DictSource(synthetic_encoder_state_dict(seed, layers))
        else:
            source = SafetensorsSource(str(checkpoint))
        self.WEIGHT_SPEC = build_encoder_spec(layers)
        WeightLoader(source, target=self, spec=self.WEIGHT_SPEC).run()
        dev = self.device
        for n in ("w_qkv", "w_o", "w_gu", "w_d"):
            setattr(self, n, getattr(self, n).view(torch.uint8).to(dev))
        for n in ("ws_qkv", "ws_o", "ws_gu", "ws_d"):
            setattr(self, n + "_t", torch.tensor(getattr(self, n), dtype=torch.float32, device=dev))
        S = max_seq
        z = lambda *shape, dtype=BF16: torch.zeros(*shape, dtype=dtype, device=dev)  # noqa: E731
        self.x, self.xn = z(S, ENC_D), z(S, ENC_D)
        self.h_bf16 = z(S, ENC_D)
        self.qkv, self.q, self.attn = z(S, QKV_N), z(S, ENC_NH * ENC_HD), z(S, ENC_NH * ENC_HD)
        self.merged, self.hidden = z(S, 2 * ENC_H), z(S, ENC_H)
        self.act8, self.attn8 = z(S, ENC_D, dtype=torch.uint8), z(S, ENC_NH * ENC_HD, dtype=torch.uint8)
        self.hid8 = z(S, ENC_H, dtype=torch.uint8)
        self.ones = torch.ones(ENC_D, dtype=BF16, device=dev)
        self.rope = rope_rows(S).to(dev)
        # scratch of the attention's key splits (the split is chosen by the prefix length)
        self.o_accum = torch.empty(ATTN_SPLITS, ENC_NH, S, ENC_HD, dtype=torch.float32, device=dev)
        self.lse_accum = torch.empty(ATTN_SPLITS, ENC_NH, S, dtype=torch.float32, device=dev)
        # partials of the down projection's K splits: one wave of CTA pairs
        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        self.splitk_ws = torch.empty(sms // 2 * 65536, dtype=torch.float32, device=dev)
        self.splitk_counters = z(8 * sms, dtype=torch.int32)
        self.attn_counters = z(2 * ((S * ENC_NH + 127) // 128), dtype=torch.int32)
        self.act_scale = torch.ones(layers, len(SITES), dtype=torch.float32, device=dev)
        self.scratch_scale = torch.zeros(1, dtype=torch.float32, device=dev)
        self.gemm = fvk.GemmRunner()
        # Addresses of what an encoder owns for its lifetime, taken once: a pass is 140 launches from Python, and indexing the
        # tensors for them took 6 of the 10 us that each one cost the host (a pass over 100 rows 1.43 ms on 1.08 ms of device time)
        buffers = ("x", "xn", "h_bf16", "qkv", "q", "attn", "merged", "hidden", "act8", "attn8", "hid8", "ones", "rope", "o_accum",
                   "lse_accum", "splitk_ws", "splitk_counters", "attn_counters", "scratch_scale")
        self._p = {n: getattr(self, n).data_ptr() for n in buffers}
        weights = ("w_qkv", "ws_qkv_t", "w_o", "ws_o_t", "w_gu", "ws_gu_t", "w_d", "ws_d_t")
        self._w = [{n: getattr(self, n)[i].data_ptr() for n in weights} for i in range(layers)]
        self._scales = [{site: self.act_scale[i, j].data_ptr() for j, site in enumerate(SITES)} for i in range(layers)]
        self.stream = torch.cuda.Stream(device=dev)
        self.stream.wait_stream(torch.cuda.current_stream(dev))       # weights, tables and buffers were written there
        self.calibrated = False

    # ------------------------------------------------------------------
    def _sp(self, layer, site):
        return self._scales[layer][site]

    def _dyn_quant(self, src, dst8, layer, site, st):
        fvk.quantize_fp8_device(src.data_ptr(), dst8.data_ptr(), self.scratch_scale.data_ptr(), src.numel(), st)
        fvk.fp8_accumulate_scale_max(self.scratch_scale.data_ptr(), self._sp(layer, site), st)
        fvk.quantize_fp8_static(src.data_ptr(), dst8.data_ptr(), self._sp(layer, site), src.numel(), st)

    def _norm(self, seq, delta, layer, site, st, calibrate):
        """(x += delta) ; RMSNorm with unit weight -> FP8 input of ``site``.  ``delta``: address or None."""
        p = self._p
        if not calibrate:
            fvk.call("frt_b200_norm_fp8", p["x"], delta, None, 0, p["ones"], None, 0, p["act8"], None, seq, ENC_D, 1e-6,
                     self._sp(layer, site), 1, st)
            return
        fvk.call("frt_b200_norm_bf16", p["x"], delta, None, 0, p["ones"], None, 0, p["h_bf16"], None, seq, ENC_D, 1e-6, 0, st)
        self._dyn_quant(self.h_bf16[:seq], self.act8[:seq], layer, site, st)

    def _gemm(self, a8, w8, ws, out, M, N, K, sp, st, pdl):
        # pdl (not while calibrating): weights, tables and scales are settled before a pass begins and may be fetched early
        self.gemm.fp8_nt_dev(a8, w8, out, M, N, K, sp, ws, st, pdl=pdl)

    def transformer_encoder(self, seq: int, k_out: torch.Tensor, v_out: torch.Tensor, st: int, calibrate: bool):
        """Runs the layers on ``self.x[:seq]``; layer i writes rows [0, seq) of k_out[i] / v_out[i] ((rows, 256))."""
        L, p, pdl = self.layers, self._p, not calibrate
        QD, KD = ENC_NH * ENC_HD, ENC_NKV * ENC_HD
        qs, ks = (seq * QD, QD, ENC_HD), (k_out.shape[1] * ENC_HD, ENC_HD, ENC_HD)
        k0, v0 = k_out.data_ptr(), v_out.data_ptr()
        k_step, v_step = k_out.stride(0) * k_out.element_size(), v_out.stride(0) * v_out.element_size()
        scale = 1.0 / math.sqrt(ENC_HD)
        for i in range(L):
            w, k, v = self._w[i], k0 + i * k_step, v0 + i * v_step
            self._norm(seq, p["xn"] if i > 0 else None, i, "qkv", st, calibrate)
            self._gemm(p["act8"], w["w_qkv"], w["ws_qkv_t"], p["qkv"], seq, QKV_N, ENC_D, self._sp(i, "qkv"), st, pdl)
            fvk.qkv_split_rope(p["qkv"], p["rope"], p["q"], k, v, seq, QD, KD, KD, ENC_HD, st, pdl=pdl)
            if i == L - 1:
                return
            if calibrate:
                fa2.fwd_bf16(p["q"], k, v, p["attn"], 0, 0, 0, 1, seq, seq, ENC_NH, ENC_NKV, ENC_HD, qs, ks, ks, qs, scale, 0, st)
                self._dyn_quant(self.attn[:seq], self.attn8[:seq], i, "o", st)
            else:
                fa2.fwd_bf16(p["q"], k, v, p["attn"], 0, p["lse_accum"], p["o_accum"], 1, seq, seq, ENC_NH, ENC_NKV, ENC_HD, qs,
                             ks, ks, qs, scale, 0, st, kv_splits=ATTN_SPLITS, flags=16, counters=p["attn_counters"], pdl=True,
                             out_fp8=p["attn8"], out_scale=self._sp(i, "o"))
            self._gemm(p["attn8"], w["w_o"], w["ws_o_t"], p["xn"], seq, ENC_D, QD, self._sp(i, "o"), st, pdl)
            self._norm(seq, p["xn"], i, "gu", st, calibrate)
            if calibrate or seq <= 64:
                self._gemm(p["act8"], w["w_gu"], w["ws_gu_t"], p["merged"], seq, 2 * ENC_H, ENC_D, self._sp(i, "gu"), st, pdl)
            if calibrate:
                fvk.gate_geglu_merged(p["merged"], p["hidden"], seq, ENC_H, st)
                self._dyn_quant(self.hidden[:seq], self.hid8[:seq], i, "d", st)
            elif seq <= 64:
                fvk.gate_geglu_merged_fp8(p["merged"], p["hid8"], seq, ENC_H, self._sp(i, "d"), st, pdl=True)
            else:               # one launch: the activation under the product's MMAs
                self.gemm.fp8_nt_dev_geglu_fp8(p["act8"], w["w_gu"], p["hid8"], seq, ENC_H, ENC_D, self._sp(i, "gu"),
                                               w["ws_gu_t"], self._sp(i, "d"), st, pdl=True)
            self.gemm.fp8_nt_dev_splitk(p["hid8"], w["w_d"], p["xn"], seq, ENC_D, ENC_H, self._sp(i, "d"), w["ws_d_t"],
                                        p["splitk_ws"], self.splitk_ws.numel() * 4, p["splitk_counters"], st, pdl=pdl)

    # ------------------------------------------------------------------
    def _check(self, embeds, k_out, v_out):
        seq = embeds.shape[0]
        if embeds.shape != (seq, ENC_D) or not 0 < seq <= self.max_seq:
            raise ValueError(f"embeds must be (seq <= {self.max_seq}, {ENC_D}), got {tuple(embeds.shape)}")
        for t in (k_out, v_out):
            if t.dim() != 3 or t.shape[0] != self.layers or t.shape[1] < seq or t.shape[2] != ENC_HD or t.dtype != BF16 \
                    or not t.is_cuda or not t[0].is_contiguous():
                raise ValueError("k_out / v_out must be bf16 CUDA tensors (layers, rows >= seq, 256) with contiguous rows")
        return seq

    def calibrate(self, embeds_list) -> None:
        """Static per-site activation scales: the max over the dynamic scales of the given sample prefixes."""
        k = torch.zeros(self.layers, self.max_seq, ENC_HD, dtype=BF16, device=self.device)
        v = torch.zeros_like(k)
        per = []
        self.stream.wait_stream(torch.cuda.current_stream(self.device))      # what still writes the samples (and k, v)
        with torch.cuda.stream(self.stream):
            for e in embeds_list:
                seq = self._check(e, k, v)
                self.act_scale.zero_()
                self.x[:seq].copy_(e.to(self.device, BF16))
                self.transformer_encoder(seq, k, v, self.stream.cuda_stream, True)
                self.stream.synchronize()
                per.append(self.act_scale.clone())
            self.act_scale.copy_(torch.stack(per).max(0).values.clamp_(min=1e-12))
        self.stream.synchronize()
        if fvk.tensor_core_status() != 0:
            raise RuntimeError("a tensor-core kernel reported a timed-out wait during calibration")
        self.calibrated = True

    def encode(self, embeds: torch.Tensor, k_out: torch.Tensor, v_out: torch.Tensor) -> int:
        """embeds (seq, 2048) -> rows [0, seq) of k_out[i], v_out[i] for every layer (K with its RoPE, in the
        interleaved feature order the decoder's Q uses).  Returns seq."""
        seq = self.enqueue(embeds, k_out, v_out)
        self.stream.synchronize()
        return seq

    def enqueue(self, embeds: torch.Tensor, k_out: torch.Tensor, v_out: torch.Tensor, after=None) -> int:
        """``encode`` without the wait on the host: the work goes to ``self.stream``, behind the current stream (and the
        stream ``after``), and the current stream waits for it."""
        if not self.calibrated:
            raise RuntimeError("calibrate() first: the encoder runs with static activation scales")
        seq = self._check(embeds, k_out, v_out)
        here = torch.cuda.current_stream(self.device)
        self.stream.wait_stream(here)
        if after is not None:
            self.stream.wait_stream(after)
        with torch.cuda.stream(self.stream):
            self.x[:seq].copy_(embeds.to(self.device, BF16), non_blocking=True)
            self.transformer_encoder(seq, k_out, v_out, self.stream.cuda_stream, False)
        here.wait_stream(self.stream)
        return seq
