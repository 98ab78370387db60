"""Wan2.2-shape video-DiT denoise step on B200, tensor-parallel over heads and FFN columns.

Block structure (the block arithmetic itself lives in the external ``wan`` package,
which the reference only wraps — ``flash_rt/frontends/torch/wan22_rtx.py:140-207`` — so this follows the
kernel call sites the reference does contain, ``flash_rt/models/motus/_fp8_swap.py:341-455`` and
``_modulate_fuse_swap.py:1-33,659-740``):

    e[0..5] = layer_modulation[6, D] + time_projection[B, 6, D]          (shift, scale, gate) x (attention, FFN)
    h   = adaLN(x; scale e1, shift e0) -> FP8 ; qkv = h W_qkv + b        (fused QKV, FP8 GEMM)
    q,k = RMSNorm over the full width (norm_q / norm_k) ; 3-D RoPE on complex pairs ; v = view
    x  += (attention(q, k, v) W_o + b_o) * e2                            (bf16 flash attention, FP8 GEMM)
    x  +=  attention(RMSNorm(LN_affine(x) W_cq + b), k_text, v_text) W_co + b_co        (cross-attention, 512 text tokens)
    x  += (gelu_tanh(adaLN(x; e4, e3) W_1 + b_1) W_2 + b_2) * e5         (FP8 GEMMs, GELU fused with the FP8 quantiser)

Tensor parallelism (the reference has none): QKV / cross-Q / W_1 are column-parallel (heads / TP, FFN / TP per
rank), W_o / W_co / W_2 row-parallel.  The residual stream is SEQUENCE-parallel: every rank keeps M / TP rows of x,
runs LayerNorm / adaLN / residual / gate on those rows only, all-gathers the FP8 producer output (1 byte per
element) in front of a column-parallel projection and reduce-scatters the bf16 partial of a row-parallel one
(half the bytes of the all-reduce it replaces, and no replicated row work).  Rows are owned in an interleaved
pattern -- block c * TP + r of M / (TP * C) rows belongs to rank r -- so that piece c of the C pieces of a tensor
is one contiguous range of rows on every rank: the collective of one piece (NCCL, side stream) runs while the
GEMM of the next piece computes.  ``sequence_parallel=False`` keeps the replicated stream with an all-reduce per
row-parallel projection.  The full-width q/k RMSNorms need the sum of squares over all heads: each rank forms its
partial (one float per row) and a tiny all-reduce completes it.  The text keys / values do not depend on the latent,
so they are projected once per prompt (``set_context``), not per step.

PyTorch provides device memory, streams and ``torch.distributed``; every arithmetic step is a kernel of this library.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from . import flash_rt_fa2 as fa2
from . import flash_rt_kernels as fvk

BF16 = torch.bfloat16
FP8 = torch.float8_e4m3fn


# ------------------------------------------------------------------ synthetic weights (full, unsharded)
def synthetic_wan_state(seed: int = 0, layers: int = 30, dim: int = 3072, ffn: int = 14336, text_dim: int = 4096,
                        head_dim: int = 128) -> dict:
    """Random-init block weights, matrices ~ N(0, 0.02) stored (out, in), biases ~ N(0, 0.02), norm weights 1."""
    g = torch.Generator().manual_seed(seed)
    w = lambda *s: torch.randn(*s, generator=g) * 0.02  # noqa: E731
    blocks = []
    for _ in range(layers):
        blocks.append({
            "modulation": w(6, dim) * 5,
            "q": w(dim, dim), "k": w(dim, dim), "v": w(dim, dim), "q_b": w(dim), "k_b": w(dim), "v_b": w(dim),
            "norm_q": torch.ones(dim), "norm_k": torch.ones(dim),
            "o": w(dim, dim), "o_b": w(dim),
            "norm3_w": torch.ones(dim), "norm3_b": torch.zeros(dim),
            "cq": w(dim, dim), "cq_b": w(dim), "ck": w(dim, text_dim), "ck_b": w(dim), "cv": w(dim, text_dim),
            "cv_b": w(dim), "norm_cq": torch.ones(dim), "norm_ck": torch.ones(dim), "co": w(dim, dim), "co_b": w(dim),
            "ffn1": w(ffn, dim), "ffn1_b": w(ffn), "ffn2": w(dim, ffn), "ffn2_b": w(dim),
        })
    return {"blocks": blocks, "dim": dim, "ffn": ffn, "text_dim": text_dim, "head_dim": head_dim}


def rope_3d_freqs(grid, head_dim: int = 128, theta: float = 10000.0):
    """(F*H*W, head_dim/2) cos and sin tables: the head's complex pairs are split between the frame, row and column
    axes (d - 4(d//6), 2(d//6), 2(d//6) real dims), each rotated by its own coordinate."""
    F, H, W = grid
    d = head_dim
    dims = (d - 4 * (d // 6), 2 * (d // 6), 2 * (d // 6))
    parts = []
    for n, dd in zip((F, H, W), dims):
        inv = 1.0 / (theta ** (np.arange(0, dd, 2, dtype=np.float64) / dd))
        parts.append(np.arange(n, dtype=np.float64)[:, None] * inv[None, :])
    f = np.broadcast_to(parts[0][:, None, None, :], (F, H, W, parts[0].shape[1]))
    h = np.broadcast_to(parts[1][None, :, None, :], (F, H, W, parts[1].shape[1]))
    ww = np.broadcast_to(parts[2][None, None, :, :], (F, H, W, parts[2].shape[1]))
    ang = np.concatenate([f, h, ww], axis=-1).reshape(F * H * W, d // 2)
    return torch.from_numpy(np.cos(ang).astype(np.float32)), torch.from_numpy(np.sin(ang).astype(np.float32))


def shard_rows(w: torch.Tensor, rank: int, tp: int) -> torch.Tensor:
    """Column-parallel layer: this rank's block of OUTPUT features (rows of an (out, in) matrix / bias entries)."""
    n = w.shape[0] // tp
    return w[rank * n:(rank + 1) * n].contiguous()


def shard_cols(w: torch.Tensor, rank: int, tp: int) -> torch.Tensor:
    """Row-parallel layer: this rank's block of INPUT features (columns of an (out, in) matrix)."""
    n = w.shape[1] // tp
    return w[:, rank * n:(rank + 1) * n].contiguous()


def _q8(w: torch.Tensor, device):
    """Per-tensor FP8 E4M3 with scale max(amax/448, 1e-12), quantised from the bf16-rounded weight."""
    wf = w.to(BF16).float()
    s = max(float(wf.abs().max()) / 448.0, 1e-12)
    return ((wf / s).clamp(-448, 448).to(FP8).view(torch.uint8).to(device),
            torch.tensor([s], dtype=torch.float32, device=device))


SITES = ("qkv", "o", "cq", "co", "f1", "f2")


# ------------------------------------------------------------------ sequence-parallel row ownership (host logic)
def sp_layout(rows: int, rows_per_batch: int, tp: int, want_pieces: int):
    """(pieces C, rows per block Mb) of the sequence-parallel residual stream, or None when the rows do not divide.
    A tensor of ``rows`` rows is cut into C pieces of tp * Mb rows; block c * tp + r (Mb rows) belongs to rank r.
    Required: whole blocks, every block inside one batch element (its modulation rows), and a piece made of whole
    batch elements or a whole fraction of one (attention may be launched per piece).  The largest C not above
    ``want_pieces`` out of (want_pieces, 4, 2, 1) that satisfies this is taken."""
    for C in (want_pieces, 4, 2, 1):
        if C < 1 or C > max(want_pieces, 1) or rows % (tp * C):
            continue
        n, mb = rows // C, rows // (tp * C)
        if rows_per_batch % mb == 0 and (n % rows_per_batch == 0 or rows_per_batch % n == 0):
            return C, mb
    return None


def sp_block_rows(c: int, rank: int, tp: int, mb: int):
    """Global rows [first, last) of rank ``rank``'s block of piece ``c``."""
    first = (c * tp + rank) * mb
    return first, first + mb


class WanDiTB200:
    def __init__(self, state: dict, *, grid=(13, 30, 52), batch: int = 2, text_len: int = 512, device=0,
                 tp_rank: int = 0, tp_size: int = 1, tp_group=None, repeat_blocks: int = 1,
                 fuse_epilogues: bool = True, overlap_chunks: int = 4, sequence_parallel: bool = True,
                 split_attention: bool = False, fast_gelu: bool = True):
        if not torch.cuda.is_available():
            raise RuntimeError("flashrt_b200 needs a CUDA device (sm_100a); there is no CPU path")
        self.device = torch.device("cuda", device)
        torch.cuda.set_device(self.device)
        self.dim, self.ffn, self.text_dim, self.hd = state["dim"], state["ffn"], state["text_dim"], state["head_dim"]
        self.heads = self.dim // self.hd
        self.tp, self.rank, self.group = tp_size, tp_rank, tp_group
        if self.heads % tp_size or self.ffn % tp_size:
            raise ValueError("heads and FFN width must divide by the tensor-parallel size")
        self.hl = self.heads // tp_size                 # local heads
        self.dl = self.hl * self.hd                     # local attention width
        self.fl = self.ffn // tp_size                   # local FFN width
        self.grid, self.B, self.T = grid, batch, text_len
        self.L = grid[0] * grid[1] * grid[2]
        self.M = self.B * self.L
        dev = self.device
        r, tp = tp_rank, tp_size
        self.blocks = []
        for bw in state["blocks"]:
            b = {}
            qkv = torch.cat([shard_rows(bw["q"], r, tp), shard_rows(bw["k"], r, tp), shard_rows(bw["v"], r, tp)], 0)
            b["qkv8"], b["qkv_s"] = _q8(qkv, dev)
            b["qkv_b"] = torch.cat([shard_rows(bw[n], r, tp) for n in ("q_b", "k_b", "v_b")]).to(dev, BF16)
            b["norm_q"], b["norm_k"] = shard_rows(bw["norm_q"], r, tp).to(dev, BF16), shard_rows(bw["norm_k"], r, tp).to(dev, BF16)
            b["o8"], b["o_s"] = _q8(shard_cols(bw["o"], r, tp), dev)
            b["cq8"], b["cq_s"] = _q8(shard_rows(bw["cq"], r, tp), dev)
            b["cq_b"] = shard_rows(bw["cq_b"], r, tp).to(dev, BF16)
            b["ck8"], b["ck_s"] = _q8(shard_rows(bw["ck"], r, tp), dev)
            b["cv8"], b["cv_s"] = _q8(shard_rows(bw["cv"], r, tp), dev)
            b["ck_b"], b["cv_b"] = shard_rows(bw["ck_b"], r, tp).to(dev, BF16), shard_rows(bw["cv_b"], r, tp).to(dev, BF16)
            b["norm_cq"], b["norm_ck"] = shard_rows(bw["norm_cq"], r, tp).to(dev, BF16), shard_rows(bw["norm_ck"], r, tp).to(dev, BF16)
            b["co8"], b["co_s"] = _q8(shard_cols(bw["co"], r, tp), dev)
            b["f18"], b["f1_s"] = _q8(shard_rows(bw["ffn1"], r, tp), dev)
            b["f1_b"] = shard_rows(bw["ffn1_b"], r, tp).to(dev, BF16)
            b["f28"], b["f2_s"] = _q8(shard_cols(bw["ffn2"], r, tp), dev)
            # biases of row-parallel layers are added once (rank 0), before the all-reduce sums the partials
            for n, src in (("o_b", "o_b"), ("co_b", "co_b"), ("f2_b", "ffn2_b")):
                b[n] = bw[src].to(dev, BF16) if r == 0 else None
            b["norm3_w"], b["norm3_b"] = bw["norm3_w"].to(dev, BF16), bw["norm3_b"].to(dev, BF16)
            b["modulation"] = bw["modulation"].to(dev, torch.float32)
            self.blocks.append(b)
        # synthetic benchmarking at full depth without generating 5 GB of random numbers on the host: every extra
        # block gets its own device copy of the weights, so that each block still streams distinct memory
        base = list(self.blocks)
        for _ in range(repeat_blocks - 1):
            for b in base:
                self.blocks.append({k: (v.clone() if isinstance(v, torch.Tensor) else v) for k, v in b.items()})
        fre, fim = rope_3d_freqs(grid, self.hd)
        self.fre, self.fim = fre.to(dev), fim.to(dev)
        M, D, dl, fl = self.M, self.dim, self.dl, self.fl
        z = lambda *s, dtype=BF16: torch.zeros(*s, dtype=dtype, device=dev)  # noqa: E731
        self.x = z(M, D)
        self.h8 = z(M, D, dtype=torch.uint8)
        self.hb = z(M, D)                                  # calibration: un-quantised producer output
        self.qkv = z(M, 3 * dl)
        self.q, self.k = z(M, dl), z(M, dl)
        self.a, self.a8 = z(M, dl), z(M, dl, dtype=torch.uint8)
        self.o = z(M, D)
        self.cq, self.cqn = z(M, dl), z(M, dl)
        self.f1, self.f8 = z(M, fl), z(M, fl, dtype=torch.uint8)
        self.ssq = z(2, M, dtype=torch.float32)
        self.e2 = z(2, 6, self.B, D)                       # modulation tensors, alternating between blocks
        self.ctx_k = self.ctx_v = None
        self.scales = torch.ones(len(self.blocks), len(SITES), dtype=torch.float32, device=dev)
        self.scratch = torch.zeros(1, dtype=torch.float32, device=dev)
        self.gemm = fvk.GemmRunner()
        self.fuse_epilogues = fuse_epilogues
        # GELU of the fused FFN-up epilogue through the hardware tanh (2^-11 relative): with the exactly rounded form the
        # epilogue of a tile outlasts its MMAs at K = 3072 (step 600 -> 580 ms on one GPU).  False: the bytes of
        # GEMM -> bias_gelu_quantize_fp8_static_bf16.
        self.fast_gelu = bool(fast_gelu)
        # row-parallel GEMM + all-reduce: the rows are cut into this many pieces so that the all-reduce of piece c
        # (NCCL, side stream) runs while the GEMM of piece c + 1 computes
        self.overlap_chunks = max(1, int(overlap_chunks)) if tp_size > 1 else 1
        self.comm_stream = torch.cuda.Stream(device=self.device) if tp_size > 1 else None
        # sequence-parallel residual stream: C pieces of tp x Mb rows; needs whole blocks of rows per rank and piece,
        # each inside one batch element (its modulation rows)
        self.sp = False
        self.split_attention = bool(split_attention)
        if tp_size > 1 and sequence_parallel:
            lay = sp_layout(M, self.L, tp_size, self.overlap_chunks)
            if lay is not None:
                self.sp, (self.C, self.Mb) = True, lay
        if self.sp:
            Ml = self.Mb * self.C
            self.xl, self.ol = z(Ml, D), z(Ml, D)
            self.h8l = z(Ml, D, dtype=torch.uint8)
        self.calibrated = False
        self.launches_per_step = 0

    # ---- helpers -------------------------------------------------------------
    def _sp(self, i, site):
        return self.scales[i, SITES.index(site)].data_ptr()

    def _allreduce(self, t):
        if self.tp > 1:
            torch.distributed.all_reduce(t, group=self.group)

    def _gemm(self, a8, w8, ws, out, M, N, K, scale_ptr, st, bias=None):
        self.gemm.fp8_nt_dev(a8.data_ptr(), w8.data_ptr(), out.data_ptr(), M, N, K, scale_ptr, ws.data_ptr(), st,
                             bias=bias.data_ptr() if bias is not None else None)
        self.launches_per_step += 1

    def _gemm_allreduce(self, a8, w8, ws, out, M, N, K, scale_ptr, st, bias=None):
        """Row-parallel projection: out = sum over ranks of (a8 . w8^T [+ bias]).  With more than one rank the rows are
        processed in pieces and each piece is all-reduced on the communication stream while the next one computes."""
        C = self.overlap_chunks
        if self.tp == 1 or C == 1 or M < getattr(self, "_min_chunk_rows", 256) * C:
            self._gemm(a8, w8, ws, out, M, N, K, scale_ptr, st, bias=bias)
            self._allreduce(out)
            return
        rows = ((M + C - 1) // C + 127) // 128 * 128
        cur = torch.cuda.current_stream()
        r0 = 0
        while r0 < M:
            r1 = min(M, r0 + rows)
            self._gemm(a8[r0:r1], w8, ws, out[r0:r1], r1 - r0, N, K, scale_ptr, st, bias=bias)
            ev = torch.cuda.Event()
            ev.record(cur)
            with torch.cuda.stream(self.comm_stream):
                self.comm_stream.wait_event(ev)
                torch.distributed.all_reduce(out[r0:r1], group=self.group)
            r0 = r1
        done = torch.cuda.Event()
        done.record(self.comm_stream)
        cur.wait_event(done)

    # ---- sequence-parallel pieces ---------------------------------------------------
    def _piece(self, t, c):
        """Rows of piece c of a full (M, ...) tensor: the blocks c * tp .. c * tp + tp - 1, one per rank."""
        n = self.tp * self.Mb
        return t[c * n:(c + 1) * n]

    def _local(self, t, c):
        """Rows of this rank's block of piece c inside a local (C * Mb, ...) tensor."""
        return t[c * self.Mb:(c + 1) * self.Mb]

    def _batch_of(self, c):
        """Batch element that this rank's block of piece c lies in."""
        return sp_block_rows(c, self.rank, self.tp, self.Mb)[0] // self.L

    def _gather_then(self, produce, consume, pending=None):
        """produce(c) writes this rank's block of piece c into ``h8l``; the block is all-gathered into ``h8`` on the
        communication stream; consume(c) (main stream) runs once piece c is complete, while piece c + 1 is in flight.
        ``pending`` = what ``_scatter_after`` returned for the projection in front: its block c is awaited and
        finished right before produce(c), so the first gather starts while later blocks are still being reduced."""
        cur = torch.cuda.current_stream()
        ready = self._gather(produce, pending)
        for c in range(self.C):
            cur.wait_event(ready[c])
            consume(c)

    def _gather(self, produce, pending=None):
        """The issuing half of ``_gather_then``: returns one event per piece (its all-gather has completed)."""
        cur = torch.cuda.current_stream()
        ready = []
        for c in range(self.C):
            if pending is not None:
                cur.wait_event(pending[0][c])
                pending[1](c)
            produce(c)
            ev = torch.cuda.Event()
            ev.record(cur)
            with torch.cuda.stream(self.comm_stream):
                self.comm_stream.wait_event(ev)
                torch.distributed.all_gather_into_tensor(self._piece(self.h8, c), self._local(self.h8l, c),
                                                         group=self.group)
                done = torch.cuda.Event()
                done.record(self.comm_stream)
            ready.append(done)
        return ready

    def _scatter_after(self, compute, finish, wait=None):
        """compute(c) (main stream; everything of piece c up to the row-parallel GEMM that writes piece c of the bf16
        partial ``o``, started once ``wait[c]`` has fired); the piece is reduce-scattered into this rank's block of
        ``ol`` on the communication stream while piece c + 1 computes.  Returns (events, finish) for ``_gather_then``
        / ``_flush``: finish(c) consumes block c once its event has fired."""
        cur = torch.cuda.current_stream()
        ready = []
        for c in range(self.C):
            if wait is not None:
                cur.wait_event(wait[c])
            compute(c)
            ev = torch.cuda.Event()
            ev.record(cur)
            with torch.cuda.stream(self.comm_stream):
                self.comm_stream.wait_event(ev)
                torch.distributed.reduce_scatter_tensor(self._local(self.ol, c), self._piece(self.o, c),
                                                        group=self.group)
                done = torch.cuda.Event()
                done.record(self.comm_stream)
            ready.append(done)
        return ready, finish

    def _flush(self, pending):
        cur = torch.cuda.current_stream()
        for c in range(self.C):
            cur.wait_event(pending[0][c])
            pending[1](c)

    def _step_sequence_parallel(self, x: torch.Tensor, tp_dev: torch.Tensor) -> torch.Tensor:
        st = torch.cuda.current_stream().cuda_stream
        B, L, M, D, dl, fl, hl, hd = self.B, self.L, self.M, self.dim, self.dl, self.fl, self.hl, self.hd
        C, Mb, n = self.C, self.Mb, self.tp * self.Mb
        xf = x.reshape(M, D)
        for c in range(C):
            g0 = (c * self.tp + self.rank) * Mb
            self._local(self.xl, c).copy_(xf[g0:g0 + Mb])
        kstr_self = (L * 3 * dl, 3 * dl, hd)
        ks = (L * dl, dl, hd)
        kc = (self.T * dl, dl, hd)
        pending = None
        # attention per piece, so that the reduce-scatter of a piece overlaps the attention of the next one: opt-in
        # (``split_attention=True``) and only where a piece is whole batch elements.  Parts of a batch element cost the
        # attention kernel more in partial waves than the overlap returns (2 GPUs, 4 pieces: 346 ms against 320 ms with
        # one attention launch per block); with whole batch elements (2 pieces) 329 ms against 326 ms on 2 GPUs.
        split_attn = self.split_attention and n % L == 0 and C > 1

        def adaln(i, site, scale_rows, shift_rows):
            def produce(c):
                bi = self._batch_of(c)
                fvk.ada_layer_norm_fp8(self._local(self.xl, c).data_ptr(), scale_rows[bi].data_ptr(),
                                       shift_rows[bi].data_ptr(), self._local(self.h8l, c).data_ptr(),
                                       self._sp(i, site), Mb, D, 1e-6, st)
            return produce

        def gated(gate_rows):
            def finish(c):
                fvk.bias_gate_mul_residual_bf16(self._local(self.xl, c).data_ptr(), self._local(self.ol, c).data_ptr(),
                                                0, gate_rows[self._batch_of(c)].data_ptr(), Mb, D, st, gate_stride=0)
            return finish

        def row_parallel(a8, w8, ws, K, site, bias, before=None):
            def compute(c):
                if before is not None:
                    before(c)
                self._gemm(self._piece(a8, c), w8, ws, self._piece(self.o, c), n, D, K, self._sp(i, site), st, bias=bias)
            return compute

        def attend(q, keys, vals, Skv, kstr, vstr, site):
            """Attention of the query rows of piece c (whole batch elements, or a part of one) against the keys of
            their batch element(s): its reduce-scatter then overlaps the attention of the next piece."""
            def run(c):
                r0 = c * n
                bi = r0 // L
                nb, sq = (n // L, L) if n >= L else (1, n)
                self._attn(q[r0:r0 + n], keys[bi], vals[bi], self.a[r0:r0 + n], self.a8[r0:r0 + n], self._sp(i, site),
                           sq, Skv, kstr, vstr, st, batch=nb)
            return run

        for i, b in enumerate(self.blocks):
            # modulation rows alternate between two buffers: the FFN gate of the block before is still pending
            e_out = [self.e2[i & 1, j] for j in range(6)]
            fvk.adaln_modulation6_bf16(tp_dev.data_ptr(), b["modulation"].data_ptr(), *[t.data_ptr() for t in e_out],
                                       B, 1, D, st)
            # ---- self-attention
            self._gather_then(adaln(i, "qkv", e_out[1], e_out[0]),
                              lambda c: self._gemm(self._piece(self.h8, c), b["qkv8"], b["qkv_s"],
                                                   self._piece(self.qkv, c), n, 3 * dl, D, self._sp(i, "qkv"), st,
                                                   bias=b["qkv_b"]), pending)
            fvk.row_sumsq(self.qkv.data_ptr(), 3 * dl, 0, dl, self.ssq[0].data_ptr(), M, st)
            fvk.row_sumsq(self.qkv.data_ptr(), 3 * dl, dl, dl, self.ssq[1].data_ptr(), M, st)
            self._allreduce(self.ssq)
            fvk.qkv_split_norm_rope_bf16(self.qkv.data_ptr(), b["norm_q"].data_ptr(), b["norm_k"].data_ptr(),
                                         self.fre.data_ptr(), self.fim.data_ptr(), self.q.data_ptr(),
                                         self.k.data_ptr(), B, L, hl, hd, L, 1e-6, st,
                                         ext_ssq_q=self.ssq[0].data_ptr(), ext_ssq_k=self.ssq[1].data_ptr(), full_dim=D)
            k_b = [self.k[j * L:] for j in range(B)]
            v_b = [self.qkv[j * L:, 2 * dl:] for j in range(B)]
            if split_attn:
                before = attend(self.q, k_b, v_b, L, ks, kstr_self, "o")
            else:
                before = None
                self._attn(self.q, self.k, self.qkv[:, 2 * dl:], self.a, self.a8, self._sp(i, "o"), L, L, ks, kstr_self, st)
            pending = self._scatter_after(row_parallel(self.a8, b["o8"], b["o_s"], dl, "o", b["o_b"], before=before),
                                          gated(e_out[2]))
            # ---- cross-attention to the text tokens
            self._gather_then(
                lambda c: fvk.call("frt_b200_layer_norm", self._local(self.xl, c).data_ptr(), b["norm3_w"].data_ptr(),
                                   b["norm3_b"].data_ptr(), None, None, 0, self._local(self.h8l, c).data_ptr(), None,
                                   self._sp(i, "cq"), Mb, D, 1e-6, 0, st),
                lambda c: self._gemm(self._piece(self.h8, c), b["cq8"], b["cq_s"], self._piece(self.cq, c), n, dl, D,
                                     self._sp(i, "cq"), st, bias=b["cq_b"]), pending)
            fvk.row_sumsq(self.cq.data_ptr(), dl, 0, dl, self.ssq[0].data_ptr(), M, st)
            self._allreduce(self.ssq[0])
            fvk.rms_norm_ext(self.cq.data_ptr(), dl, b["norm_cq"].data_ptr(), self.ssq[0].data_ptr(),
                             self.cqn.data_ptr(), dl, M, dl, D, 1e-6, st)
            ck_b = [self.ctx_k[i][j * self.T:] for j in range(B)]
            cv_b = [self.ctx_v[i][j * self.T:] for j in range(B)]
            if split_attn:
                before = attend(self.cqn, ck_b, cv_b, self.T, kc, kc, "co")
            else:
                before = None
                self._attn(self.cqn, self.ctx_k[i], self.ctx_v[i], self.a, self.a8, self._sp(i, "co"), L, self.T, kc, kc,
                           st)
            pending = self._scatter_after(row_parallel(self.a8, b["co8"], b["co_s"], dl, "co", b["co_b"], before=before),
                                          lambda c: fvk.residual_add(self._local(self.xl, c).data_ptr(),
                                                                     self._local(self.ol, c).data_ptr(), Mb * D, st))
            # ---- FFN
            fused = self.fuse_epilogues and n > 256 and fl >= 128

            def ffn_up(c):
                if fused:
                    self.gemm.fp8_nt_dev_bias_gelu_fp8(self._piece(self.h8, c).data_ptr(), b["f18"].data_ptr(),
                                                       self._piece(self.f8, c).data_ptr(), n, fl, D, self._sp(i, "f1"),
                                                       b["f1_s"].data_ptr(), b["f1_b"].data_ptr(), self._sp(i, "f2"), st,
                                                       fast_gelu=self.fast_gelu)
                    self.launches_per_step += 1
                else:
                    self._gemm(self._piece(self.h8, c), b["f18"], b["f1_s"], self._piece(self.f1, c), n, fl, D,
                               self._sp(i, "f1"), st)
                    fvk.bias_gelu_quantize_fp8_static_bf16(self._piece(self.f1, c).data_ptr(), b["f1_b"].data_ptr(),
                                                           self._piece(self.f8, c).data_ptr(), self._sp(i, "f2"), n, fl, st)
            # FFN-up of every piece, then FFN-down of every piece (running the two GEMMs of a piece back to back, so that its
            # reduce-scatter overlaps both GEMMs of the next piece, measured slower: 326 against 320 ms on 2 GPUs)
            self._gather_then(adaln(i, "f1", e_out[4], e_out[3]), ffn_up, pending)
            pending = self._scatter_after(row_parallel(self.f8, b["f28"], b["f2_s"], fl, "f2", b["f2_b"]),
                                          gated(e_out[5]))
        self._flush(pending)
        # the updated tokens, gathered once per step
        out = torch.empty(M, D, dtype=BF16, device=self.device)
        for c in range(C):
            torch.distributed.all_gather_into_tensor(self._piece(out, c), self._local(self.xl, c).contiguous(),
                                                     group=self.group)
        return out.reshape(B, L, D)

    def _attn(self, q, k, v, out, out8, scale_ptr, Sq, Skv, kstr, vstr, st, batch=None):
        hl, hd = self.hl, self.hd
        qs = (Sq * hl * hd, hl * hd, hd)
        fa2.fwd_bf16(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 0, 0, 0,
                     self.B if batch is None else batch, Sq, Skv, hl, hl, hd,
                     qs, kstr, vstr, qs, 1.0 / math.sqrt(hd), 148, st,
                     out_fp8=out8.data_ptr() if scale_ptr else 0, out_scale=scale_ptr or 0)
        self.launches_per_step += 1

    def _quant_measured(self, src, dst8, i, site, st):
        """FP8 quantisation of a bf16 activation with the site's scale, measured first."""
        fvk.quantize_fp8_device(src.data_ptr(), dst8.data_ptr(), self.scratch.data_ptr(), src.numel(), st)
        fvk.fp8_accumulate_scale_max(self.scratch.data_ptr(), self._sp(i, site), st)
        fvk.quantize_fp8_static(src.data_ptr(), dst8.data_ptr(), self._sp(i, site), src.numel(), st)

    # ---- text context: projected once per prompt -------------------------------
    def set_context(self, context: torch.Tensor) -> None:
        """context (B, text_len, text_dim): per block k = RMSNorm(ctx W_ck + b), v = ctx W_cv + b for the local heads."""
        dev, B, T, dl = self.device, self.B, self.T, self.dl
        st = torch.cuda.current_stream().cuda_stream
        ctx = context.to(dev, BF16).reshape(B * T, self.text_dim).contiguous()
        c8 = torch.zeros(B * T, self.text_dim, dtype=torch.uint8, device=dev)
        cs = torch.zeros(1, dtype=torch.float32, device=dev)
        fvk.quantize_fp8_device(ctx.data_ptr(), c8.data_ptr(), cs.data_ptr(), ctx.numel(), st)
        self.ctx_k, self.ctx_v = [], []
        ssq = torch.zeros(B * T, dtype=torch.float32, device=dev)
        for b in self.blocks:
            kk = torch.zeros(B * T, dl, dtype=BF16, device=dev)
            vv = torch.zeros(B * T, dl, dtype=BF16, device=dev)
            self.gemm.fp8_nt_dev(c8.data_ptr(), b["ck8"].data_ptr(), kk.data_ptr(), B * T, dl, self.text_dim,
                                 cs.data_ptr(), b["ck_s"].data_ptr(), st, bias=b["ck_b"].data_ptr())
            self.gemm.fp8_nt_dev(c8.data_ptr(), b["cv8"].data_ptr(), vv.data_ptr(), B * T, dl, self.text_dim,
                                 cs.data_ptr(), b["cv_s"].data_ptr(), st, bias=b["cv_b"].data_ptr())
            fvk.row_sumsq(kk.data_ptr(), dl, 0, dl, ssq.data_ptr(), B * T, st)
            self._allreduce(ssq)
            kn = torch.zeros_like(kk)
            fvk.rms_norm_ext(kk.data_ptr(), dl, b["norm_ck"].data_ptr(), ssq.data_ptr(), kn.data_ptr(), dl, B * T, dl,
                             self.dim, 1e-6, st)
            self.ctx_k.append(kn)
            self.ctx_v.append(vv)
        torch.cuda.synchronize(dev)

    # ---- one denoise step -----------------------------------------------------------
    def step(self, x: torch.Tensor, time_proj: torch.Tensor, calibrate: bool = False) -> torch.Tensor:
        """x (B, L, D) latent tokens, time_proj (B, 6, D) fp32 -> updated tokens (B, L, D) bf16 (all blocks)."""
        self.launches_per_step = 0
        tp_dev = time_proj.to(self.device, torch.float32).reshape(self.B, 1, 6, self.dim).contiguous()
        x = x.to(self.device, BF16)
        if calibrate:
            return self._step_calibrate(x, tp_dev)
        return self._step_sequence_parallel(x, tp_dev) if self.sp else self._step_replicated(x, tp_dev)

    def _modulation(self, i, tp_dev, st):
        """Six (B, D) modulation tensors of block i; two sets alternate (the FFN gate of block i is read by the launch that
        also normalises for block i + 1)."""
        e = self.e2[i & 1]
        fvk.adaln_modulation6_bf16(tp_dev.data_ptr(), self.blocks[i]["modulation"].data_ptr(),
                                   *[e[j].data_ptr() for j in range(6)], self.B, 1, self.dim, st)
        return e

    def _self_attention_inputs(self, b, st):
        """Full-width q / k RMSNorm and 3-D RoPE of the packed QKV rows."""
        B, L, M, dl = self.B, self.L, self.M, self.dl
        ext = {}
        if self.tp > 1:
            fvk.row_sumsq(self.qkv.data_ptr(), 3 * dl, 0, dl, self.ssq[0].data_ptr(), M, st)
            fvk.row_sumsq(self.qkv.data_ptr(), 3 * dl, dl, dl, self.ssq[1].data_ptr(), M, st)
            self._allreduce(self.ssq)
            ext = dict(ext_ssq_q=self.ssq[0].data_ptr(), ext_ssq_k=self.ssq[1].data_ptr(), full_dim=self.dim)
        fvk.qkv_split_norm_rope_bf16(self.qkv.data_ptr(), b["norm_q"].data_ptr(), b["norm_k"].data_ptr(),
                                     self.fre.data_ptr(), self.fim.data_ptr(), self.q.data_ptr(), self.k.data_ptr(), B, L,
                                     self.hl, self.hd, L, 1e-6, st, **ext)

    def _cross_query_norm(self, b, st):
        """Full-width RMSNorm of the cross-attention queries (one pass when this rank holds all heads)."""
        M, D, dl = self.M, self.dim, self.dl
        if self.tp == 1:
            fvk.rms_norm(self.cq.data_ptr(), b["norm_cq"].data_ptr(), self.cqn.data_ptr(), M, D, 1e-6, st)
            return
        fvk.row_sumsq(self.cq.data_ptr(), dl, 0, dl, self.ssq[0].data_ptr(), M, st)
        self._allreduce(self.ssq[0])
        fvk.rms_norm_ext(self.cq.data_ptr(), dl, b["norm_cq"].data_ptr(), self.ssq[0].data_ptr(), self.cqn.data_ptr(), dl,
                         M, dl, D, 1e-6, st)

    def _step_replicated(self, x, tp_dev):
        """The residual stream in one piece on every rank.  A residual update and the LayerNorm behind it are one launch
        over all batch elements; the stream is read from the caller's ``x`` until its first update and its last update
        goes straight into the returned tensor."""
        st = torch.cuda.current_stream().cuda_stream
        L, M, D, dl, fl = self.L, self.M, self.dim, self.dl, self.fl
        ks, kv, kc = (L * dl, dl, self.hd), (L * 3 * dl, 3 * dl, self.hd), (self.T * dl, dl, self.hd)
        v_view = self.qkv[:, 2 * dl:]
        xin = x.reshape(M, D).contiguous()
        out = torch.empty(M, D, dtype=BF16, device=self.device)
        e = self._modulation(0, tp_dev, st)
        fvk.residual_layer_norm_fp8(xin.data_ptr(), 0, 0, 0, self.h8.data_ptr(), self._sp(0, "qkv"), M, D, 1e-6, st,
                                    scale=e[1].data_ptr(), shift=e[0].data_ptr(), mod_stride=D, mod_rows=L)
        res, cur = xin.data_ptr(), self.x.data_ptr()
        last = len(self.blocks) - 1
        for i, b in enumerate(self.blocks):
            # ---- self-attention
            self._gemm(self.h8, b["qkv8"], b["qkv_s"], self.qkv, M, 3 * dl, D, self._sp(i, "qkv"), st, bias=b["qkv_b"])
            self._self_attention_inputs(b, st)
            self._attn(self.q, self.k, v_view, self.a, self.a8, self._sp(i, "o"), L, L, ks, kv, st)
            self._gemm_allreduce(self.a8, b["o8"], b["o_s"], self.o, M, D, dl, self._sp(i, "o"), st, bias=b["o_b"])
            # ---- cross-attention to the text tokens
            fvk.residual_layer_norm_fp8(res, self.o.data_ptr(), e[2].data_ptr(), cur, self.h8.data_ptr(), self._sp(i, "cq"),
                                        M, D, 1e-6, st, weight=b["norm3_w"].data_ptr(), bias=b["norm3_b"].data_ptr(),
                                        mod_stride=D, mod_rows=L)
            res = cur
            self._gemm(self.h8, b["cq8"], b["cq_s"], self.cq, M, dl, D, self._sp(i, "cq"), st, bias=b["cq_b"])
            self._cross_query_norm(b, st)
            self._attn(self.cqn, self.ctx_k[i], self.ctx_v[i], self.a, self.a8, self._sp(i, "co"), L, self.T, kc, kc, st)
            self._gemm_allreduce(self.a8, b["co8"], b["co_s"], self.o, M, D, dl, self._sp(i, "co"), st, bias=b["co_b"])
            # ---- FFN
            fvk.residual_layer_norm_fp8(cur, self.o.data_ptr(), 0, cur, self.h8.data_ptr(), self._sp(i, "f1"), M, D, 1e-6,
                                        st, scale=e[4].data_ptr(), shift=e[3].data_ptr(), mod_stride=D, mod_rows=L)
            if not self.fuse_epilogues or M <= 256 or fl < 128:
                self._gemm(self.h8, b["f18"], b["f1_s"], self.f1, M, fl, D, self._sp(i, "f1"), st)
                fvk.bias_gelu_quantize_fp8_static_bf16(self.f1.data_ptr(), b["f1_b"].data_ptr(), self.f8.data_ptr(),
                                                       self._sp(i, "f2"), M, fl, st)
            else:
                # FFN-up projection with bias + GELU + FP8 quantise in the GEMM epilogue (same bytes, one launch)
                self.gemm.fp8_nt_dev_bias_gelu_fp8(self.h8.data_ptr(), b["f18"].data_ptr(), self.f8.data_ptr(), M, fl,
                                                   D, self._sp(i, "f1"), b["f1_s"].data_ptr(), b["f1_b"].data_ptr(),
                                                   self._sp(i, "f2"), st, fast_gelu=self.fast_gelu)
                self.launches_per_step += 1
            self._gemm_allreduce(self.f8, b["f28"], b["f2_s"], self.o, M, D, fl, self._sp(i, "f2"), st, bias=b["f2_b"])
            gate = e[5].data_ptr()
            if i == last:
                fvk.residual_layer_norm_fp8(cur, self.o.data_ptr(), gate, out.data_ptr(), 0, 0, M, D, 1e-6, st,
                                            mod_stride=D, mod_rows=L)
            else:
                e = self._modulation(i + 1, tp_dev, st)
                fvk.residual_layer_norm_fp8(cur, self.o.data_ptr(), gate, cur, self.h8.data_ptr(), self._sp(i + 1, "qkv"),
                                            M, D, 1e-6, st, scale=e[1].data_ptr(), shift=e[0].data_ptr(), mod_stride=D,
                                            mod_rows=L)
        return out.reshape(self.B, L, D)

    def _step_calibrate(self, x, tp_dev):
        """The step with every FP8 input produced in bf16 first and its scale measured."""
        st = torch.cuda.current_stream().cuda_stream
        L, M, D, dl, fl = self.L, self.M, self.dim, self.dl, self.fl
        ks, kv, kc = (L * dl, dl, self.hd), (L * 3 * dl, 3 * dl, self.hd), (self.T * dl, dl, self.hd)
        self.x.copy_(x.reshape(M, D))
        for i, b in enumerate(self.blocks):
            e_out = self._modulation(i, tp_dev, st)
            self._adaln_measured(i, "qkv", e_out[1], e_out[0], st)
            self._gemm(self.h8, b["qkv8"], b["qkv_s"], self.qkv, M, 3 * dl, D, self._sp(i, "qkv"), st, bias=b["qkv_b"])
            self._self_attention_inputs(b, st)
            self._attn(self.q, self.k, self.qkv[:, 2 * dl:], self.a, self.a8, 0, L, L, ks, kv, st)
            self._quant_measured(self.a, self.a8, i, "o", st)
            self._gemm_allreduce(self.a8, b["o8"], b["o_s"], self.o, M, D, dl, self._sp(i, "o"), st, bias=b["o_b"])
            self._gated_residual(self.o, e_out[2], st)
            fvk.layer_norm(self.x.data_ptr(), b["norm3_w"].data_ptr(), b["norm3_b"].data_ptr(), self.hb.data_ptr(), M, D,
                           1e-6, st)
            self._quant_measured(self.hb, self.h8, i, "cq", st)
            self._gemm(self.h8, b["cq8"], b["cq_s"], self.cq, M, dl, D, self._sp(i, "cq"), st, bias=b["cq_b"])
            self._cross_query_norm(b, st)
            self._attn(self.cqn, self.ctx_k[i], self.ctx_v[i], self.a, self.a8, 0, L, self.T, kc, kc, st)
            self._quant_measured(self.a, self.a8, i, "co", st)
            self._gemm_allreduce(self.a8, b["co8"], b["co_s"], self.o, M, D, dl, self._sp(i, "co"), st, bias=b["co_b"])
            fvk.residual_add(self.x.data_ptr(), self.o.data_ptr(), M * D, st)
            self._adaln_measured(i, "f1", e_out[4], e_out[3], st)
            self._gemm(self.h8, b["f18"], b["f1_s"], self.f1, M, fl, D, self._sp(i, "f1"), st)
            # scale of the GELU output, measured on a bf16 copy (host-side torch math)
            tmp = self.f1.clone()
            fvk.add_bias_bf16(tmp.data_ptr(), b["f1_b"].data_ptr(), M, fl, st)
            act = torch.nn.functional.gelu(tmp.float(), approximate="tanh").to(BF16)
            self._quant_measured(act, self.f8, i, "f2", st)
            fvk.bias_gelu_quantize_fp8_static_bf16(self.f1.data_ptr(), b["f1_b"].data_ptr(), self.f8.data_ptr(),
                                                   self._sp(i, "f2"), M, fl, st)
            self._gemm_allreduce(self.f8, b["f28"], b["f2_s"], self.o, M, D, fl, self._sp(i, "f2"), st, bias=b["f2_b"])
            self._gated_residual(self.o, e_out[5], st)
        return self.x.reshape(self.B, L, D).clone()

    def _adaln_measured(self, i, site, scale_rows, shift_rows, st):
        """adaLN of every batch element with its own (D,) scale / shift row, measured and quantised for ``site``."""
        L, D = self.L, self.dim
        for bi in range(self.B):
            rows = slice(bi * L, (bi + 1) * L)
            fvk.ada_layer_norm_bf16(self.x[rows].data_ptr(), scale_rows[bi].data_ptr(), shift_rows[bi].data_ptr(),
                                    self.hb[rows].data_ptr(), L, D, 1e-6, st)
        self._quant_measured(self.hb, self.h8, i, site, st)

    def _gated_residual(self, y, gate_rows, st):
        L, D = self.L, self.dim
        for bi in range(self.B):
            fvk.bias_gate_mul_residual_bf16(self.x[bi * L:(bi + 1) * L].data_ptr(), y[bi * L:(bi + 1) * L].data_ptr(),
                                            0, gate_rows[bi].data_ptr(), L, D, st, gate_stride=0)

    def calibrate(self, x: torch.Tensor, time_proj: torch.Tensor) -> None:
        """One eager pass that measures the per-site activation scales (amax / 448).  It runs on the replicated
        residual stream (all-reduce form) also when the timed step is sequence-parallel: the scales of replicated
        activations then agree across ranks by construction, those of head- / column-sharded ones are local."""
        self.scales.zero_()
        self.step(x, time_proj, calibrate=True)
        self.scales.clamp_(min=1e-12)
        torch.cuda.synchronize(self.device)
        self.calibrated = True
