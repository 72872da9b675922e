"""Native many-token forward: prompt processing and large-batch decode built from this package's
kernels only — RMSNorm, tcgen05 GEMMs (bf16 or Q4 dequantised in the main loop), RoPE + paged KV
write, paged flash attention (causal prefill kernel or split-KV decode kernel), and for MoE layers
top-k routing, row scatter, two grouped tensor-core GEMMs with SwiGLU, and the weighted combine.

``NativePrefill`` is the counterpart of ``TransformerModel::forward_prefill_graph``
(crates/rmlx-nn/src/transformer.rs:4416-4620), which encodes the 9 dispatches of a prefill layer
into shared command buffers. ``BatchedDecode`` serves decode batches beyond what the mat-vec
kernels take (more than 4 rows): one token of each of B sequences per step, every shape static, so
the whole step is captured in a CUDA graph (the reference's batched decode goes through the same
GEMM kernels with M = batch, crates/rmlx-nn/src/transformer.rs:4250-4402).

With tensor parallelism the row-parallel projections use the GEMM whose all-reduce runs inside the
kernel (``parallel.tp_gemm``) when a ``gemm_comm`` is attached to the model; the MoE block's partial
sums go through the injected ``allreduce``.
"""
from __future__ import annotations

import array
import ctypes
import os
from typing import List, Optional, Sequence

import torch

from .. import _lib
from ..kv.paged import PagedKvCache
from ..ops import decode as D
from ..ops import narrow
from ..runtime.graph import GraphCache, bucket_for
from ..ops.attention import few_rows_attention, few_rows_plan, flash_prefill_paged, prefill_kernel_choice
from ..ops.gemm import GemmStatus, gemm_bf16
from ..ops import grouped
from ..ops.grouped import moe_prefill_ffn
from ..ops.quantized import pair_pays, qmm, row_gemm, row_supported, row_tables_ready, tiles_route, xgemm
from ..ops.weights import LinearWeight, W_BF16, W_Q4, W_Q8
from .prefill_plan import PrefillPlan, prompt_offsets


def _narrow(x: torch.Tensor, w: LinearWeight) -> bool:
    """Whether these few rows go through the weight-streaming kernel (``ops/narrow.py``)."""
    return x.shape[0] <= 64 and narrow.pays(w, x.shape[0]) and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0


def _mm(x: torch.Tensor, w: LinearWeight, residual: Optional[torch.Tensor] = None) -> torch.Tensor:
    if w.kind == W_BF16:
        if _narrow(x, w) and (residual is None or narrow.same_layout(residual, None, x.shape[0], w.n)):
            return narrow.narrow_gemm(x, w, residual=residual)
        if x.shape[0] > 128 and w.w.is_contiguous() and pair_pays(W_BF16, x.shape[0], w.n, w.k):
            return xgemm(x, w, residual=residual)         # SM pairs
        return gemm_bf16(x, w.w, residual=residual)
    return qmm(x, w, residual=residual)


def _norm_fits(x: torch.Tensor, w: LinearWeight, norm: torch.Tensor) -> bool:
    """Whether ``_narrow`` rows can take their norm along (16-bit weights then use twice the tiles of rows)."""
    return _narrow(x, w) and norm.data_ptr() % 16 == 0 and (w.kind != W_BF16 or x.shape[0] <= 8)


def _norm_mm(h: torch.Tensor, norm: torch.Tensor, eps: float, w: LinearWeight) -> torch.Tensor:
    """rmsnorm(h) W^T; one launch where the weight-streaming kernel takes the rows."""
    if _norm_fits(h, w, norm):
        return narrow.narrow_gemm(h, w, norm, eps)
    return _mm(D.rms_norm(h, norm, eps), w)


def _norm_gate_up_act(h: torch.Tensor, norm: torch.Tensor, eps: float, w: LinearWeight) -> torch.Tensor:
    if w.n % 32 == 0 and _norm_fits(h, w, norm):
        return narrow.narrow_gemm(h, w, norm, eps, swiglu=True)
    return _gate_up_act(D.rms_norm(h, norm, eps), w)


def _gate_up_act(x: torch.Tensor, w: LinearWeight) -> torch.Tensor:
    """silu(x W_gate^T) * (x W_up^T) for W = [gate; up]: SwiGLU runs in the GEMM epilogue when the
    shape allows, else GEMM then the element-wise kernel."""
    if w.n % 32 == 0 and _narrow(x, w):
        return narrow.narrow_gemm(x, w, swiglu=True)
    q4_ok = w.kind == W_BF16 or (w.kind == W_Q4 and not w.scales_f16 and
                                 bool(_lib.cuda().rmlx_qgemm_supported(w.k)))
    if w.n % 256 == 0 and w.k % 8 == 0 and q4_ok:
        return xgemm(x, w, swiglu=True)
    return D.silu_mul(_mm(x, w))


def _router_logits(xn: torch.Tensor, router: torch.Tensor) -> torch.Tensor:
    """fp32 router logits from bf16 operands on this package's tensor-core GEMM, the accumulator
    stored unrounded (a bf16 result would create ties between experts)."""
    if xn.dtype == torch.bfloat16 and router.dtype == torch.bfloat16 and xn.shape[1] % 8 == 0:
        from ..ops.gemm import gemm_bf16_f32
        return gemm_bf16_f32(xn.contiguous(), router)
    return xn.float() @ router.float().t()


# Rows up to which the decode step's router (one launch from the rows before their norm) is faster than a norm, a GEMM and the
# selection: 128 experts of 4096, us, 7.4 / 26 at 64 rows, 14 / 26 at 128, 16 / 27 at 192, 23 / 27 at 256; 256 experts 26 / 28 at 192,
# 38 / 28 at 256.
ROUTER_ROWS = 192


def _logits_by_rows(w: LinearWeight, rows: int) -> bool:
    """Whether the logits of several rows come from the kernel whose product rows are the vocabulary's (``row_gemm``, fp32 unrounded), rather
    than as any projection and then converted.

    Measured (us, there / as a projection), 4-bit: 151936 x 4096 145 / 167 at 64 rows, 190 / 292 at 160; 32000 x 2048 25 / 30, 35 / 46; 50304 x 1024
    24 / 33, 41 / 49; above, two passes: at 192 rows 32768 x 4096 72 / 69, 128256 x 8192 451 / 429. Small vocabularies, which the tiles
    hold in one round, and short K up to 64 rows: 8192 x 2048 18 / 19 at 64, 22 / 19 at 96; 2048 x 1024 12.5 / 13.3, 13.7 / 13.5, at 160 17.5 / 13.5;
    65536 x 512 25 / 27 at 64, 37 / 34 at 112."""
    return w.kind == W_Q4 and rows <= (160 if w.n >= 16384 and w.k >= 1024 else 64)


def _routed_few(h: torch.Tensor, lw, moe) -> bool:
    """Whether few rows go to the experts without a normalised copy of them: the router and the weight-streaming kernel take the norm
    along."""
    up, r = lw.experts_gate_up, lw.router
    return (h.shape[0] <= ROUTER_ROWS and up.experts == moe.num_experts and not lw.expert_base and grouped._NARROW_MAX_AVG_ROWS <= 0 and
            narrow.pays_grouped(up, lw.experts_down, h.shape[0] * moe.num_experts_per_token) and r.dtype == torch.bfloat16 and
            r.is_contiguous() and h.stride(0) % 8 == 0 and (h.data_ptr() | r.data_ptr() | lw.norm2.data_ptr()) % 16 == 0)


def _check_model(model) -> None:
    cfg = model.cfg
    if cfg.head_dim not in (64, 128):
        raise ImportError("the native forward covers head_dim 64 and 128")
    if model.w.embed.dtype != torch.bfloat16:
        raise ImportError("the native forward needs bf16 activations")


class _Layers:
    """The per-layer body shared by prefill and batched decode; ``attend`` does RoPE, the KV write
    and attention for the caller's token layout."""

    def __init__(self, model):
        _check_model(model)
        self.m = model
        self.comm = getattr(model, "gemm_comm", None)

    def _row_parallel(self, x: torch.Tensor, w: LinearWeight, h: torch.Tensor) -> torch.Tensor:
        m = self.m
        if m.layout.world == 1:
            return _mm(x, w, residual=h)
        if self.comm is not None:
            return self.comm.gemm_allreduce(x, w, residual=h.contiguous())
        return h + m._sum(_mm(x, w))

    def run(self, h: torch.Tensor, attend) -> torch.Tensor:
        m = self.m
        cfg, w = m.cfg, m.w
        t = h.shape[0]
        hd, hq = cfg.head_dim, m.hq
        for li, lw in enumerate(w.layers):
            qkv = _norm_mm(h, lw.norm1, cfg.rms_norm_eps, lw.wqkv)
            attn = attend(li, qkv)
            h = self._row_parallel(attn.view(t, hq * hd), lw.wo, h)
            if lw.router is not None:
                moe = cfg.ff_type.moe
                single = m.layout.world == 1 and lw.shared_gate_up is None
                if single and _routed_few(h, lw, moe):
                    idx, wts = D.moe_router(h, lw.router, lw.norm2, cfg.rms_norm_eps, moe.num_experts_per_token, lw.expert_bias)
                    h = narrow.expert_ffn(h, idx, wts, lw.experts_gate_up, lw.experts_down, lw.norm2, cfg.rms_norm_eps, residual=h)
                    continue
                xn = D.rms_norm(h, lw.norm2, cfg.rms_norm_eps)
                logits = _router_logits(xn, lw.router)
                idx, wts, _, offsets = D.topk_route(logits, moe.num_experts_per_token, lw.expert_bias)
                y = moe_prefill_ffn(xn, idx, wts, offsets, lw.experts_gate_up, lw.experts_down,
                                    residual=h if single else None, expert_base=lw.expert_base)
                if lw.shared_gate_up is not None:
                    y = y + _mm(_gate_up_act(xn, lw.shared_gate_up), lw.shared_down)
                h = y if single else h + m._sum(y)
            else:
                act = _norm_gate_up_act(h, lw.norm2, cfg.rms_norm_eps, lw.w_gate_up)
                h = self._row_parallel(act, lw.w_down, h)
        return h

    def logits(self, rows: torch.Tensor) -> torch.Tensor:
        """Final norm + LM head for a few rows [R, D] -> fp32 [R, vocab] (gathered over TP ranks)."""
        m = self.m
        cfg, w = m.cfg, m.w
        r = rows.shape[0]
        rows = rows.contiguous()
        # more rows than the per-row kernels are for only if rms_gemv will take the weight-streaming kernel
        if r <= 4 or (narrow.pays(w.lm_head, r) and D._several(r, w.lm_head, rows, w.final_norm)):
            out = D.rms_gemv(rows, w.lm_head, w.final_norm, cfg.rms_norm_eps,
                             out=torch.empty(r, w.lm_head.n, dtype=torch.float32, device=m.device))
        else:
            xn = D.rms_norm(rows, w.final_norm, cfg.rms_norm_eps)
            if w.lm_head.kind == W_BF16 and w.lm_head.k % 8 == 0:
                from ..ops.gemm import gemm_bf16_f32       # accumulator stored unrounded
                out = gemm_bf16_f32(xn, w.lm_head.w)
            elif _logits_by_rows(w.lm_head, r) and row_supported(
                    xn, w.lm_head, out := torch.empty(r, w.lm_head.n, dtype=torch.float32, device=m.device)):
                row_gemm(xn, w.lm_head, out=out)
            else:
                out = _mm(xn, w.lm_head).float()
        if m.allgather_logits is not None and m.layout.world > 1 and w.lm_head.n != cfg.vocab_size:
            out = m.allgather_logits(out)
        return out


_lib.register_cuda_sigs({
    "rmlx_prompt_sizes": ("p", "i"),
    "rmlx_prompt_run": ("ppffppp", "i"),
})


class PromptRun:
    """A prompt portion from one native call (csrc/runtime/prompt_run.cu): the launches of ``_Layers.run`` with the kernels that it
    would choose, without the interpreter between them. Pointers, sizes and choices are taken from the model and the cache at every call;
    kept are only the two tables of numbers. ``run`` returns None for what it does not cover (tensor parallelism, shared experts, weights
    at odd addresses, one launch at a time for debugging): the caller then goes launch by launch."""

    NARROW, ROW, PAIR, TILES, BF16, EXPAND, WITH_NORM, SWIGLU = 1, 2, 3, 4, 5, 6, 16, 32

    def __init__(self, model):
        self.m = model
        self._words: tuple = ()             # 64-bit words of the native call's two records
        self._numbers: list = []            # int32 0, 1, 2, ... and zeros on the device; grown ones are kept beside their successors
        if model.layout.world == 1 and model.device.type == "cuda":
            self._tables(model.cfg.max_seq_len + 1)     # here, not in the first portion that needs them

    def _tables(self, n: int):
        if not self._numbers or self._numbers[-1][0].numel() < n:
            size = max(n, 2 * self._numbers[-1][0].numel() if self._numbers else 0)
            dev = self.m.device
            pair = (torch.arange(size, dtype=torch.int32, device=dev), torch.zeros(size, dtype=torch.int32, device=dev))
            torch.cuda.current_stream(dev).synchronize()    # from here on any stream may read them
            self._numbers.append(pair)
        return self._numbers[-1]

    # ------------------------------------------------------------------ routes
    def _plain(self, w: LinearWeight, t: int) -> int:
        """What ``_mm`` does with rows on 16 bytes; 0: not covered."""
        if t <= 64 and narrow.pays(w, t):
            return self.NARROW
        if w.kind == W_BF16:
            if not w.w.is_contiguous() or w.w.dtype != torch.bfloat16:
                return 0
            return self.PAIR if t > 128 and pair_pays(W_BF16, t, w.n, w.k) and tiles_route(w, t) == "pair" else self.BF16
        if w.kind == W_Q4 and not w.scales_f16 and w.k % 512 == 0:
            return self._tiles(w, t)
        return self.EXPAND

    def _tiles(self, w: LinearWeight, t: int, experts: int = 0, swiglu: bool = False) -> int:
        route = tiles_route(w, t, experts, swiglu)
        if route == "row" and not row_tables_ready(w):
            route = tiles_route(w, t, experts, swiglu, row=False)
        return {"row": self.ROW, "pair": self.PAIR, "tiles": self.TILES}[route]

    def _normed(self, w: LinearWeight, t: int, norm: torch.Tensor) -> int:
        route = self._plain(w, t)
        return route | self.WITH_NORM if route == self.NARROW and norm.data_ptr() % 16 == 0 and (w.kind != W_BF16 or t <= 8) else route

    def _gate_up(self, w: LinearWeight, t: int, norm: torch.Tensor) -> int:
        route = self._normed(w, t, norm)
        if route & 15 == self.NARROW:
            return route | self.SWIGLU if w.n % 32 == 0 else route & 15
        if w.n % 256 == 0 and w.k % 8 == 0 and (w.kind == W_BF16 or (w.kind == W_Q4 and not w.scales_f16 and w.k % 512 == 0)):
            return 0 if not w.w.is_contiguous() else self._tiles(w, t, swiglu=True) | self.SWIGLU
        return route

    # ------------------------------------------------------------------ the pass
    def run(self, token_ids: torch.Tensor, cache: PagedKvCache, seq_id: int, pos0: int) -> Optional[torch.Tensor]:
        m = self.m
        cfg, mw = m.cfg, m.w
        t, d, hd, hq, hkv = token_ids.numel(), cfg.hidden_size, cfg.head_dim, m.hq, m.hkv
        if m.layout.world != 1 or _lib.debug_serialize() or grouped._NARROW_MAX_AVG_ROWS > 0 or d % 64 or cache.block_size != 16 or \
                token_ids.dtype != torch.int32 or not token_ids.is_contiguous() or not mw.embed.is_contiguous():
            return None
        bf16, pages = torch.bfloat16, (pos0 + t + 15) // 16
        q8 = cache.quantized
        row = cache.block_table[cache.slot_of[seq_id]]
        # addresses go to the kernels unseen: host tensors, and ids of another device, are left to the launches one by one, which raise
        if not mw.embed.is_cuda or not m.cos.is_cuda or not token_ids.device == row.device == mw.embed.device:
            return None
        if row.numel() < pages or mw.embed.dtype != bf16:
            return None
        recs = array.array("q")
        mid = act = dense = xs = y = pairs = most = 0
        for li, lw in enumerate(mw.layers):
            n1, n2, kc, vc = lw.norm1, lw.norm2, cache.k[li], cache.v[li]
            p1, p2 = n1.data_ptr(), n2.data_ptr()
            if n1.dtype != bf16 or n2.dtype != bf16 or (p1 | p2) % 16 or not n1.is_contiguous() or not n2.is_contiguous() \
                    or not kc.is_contiguous() or not vc.is_contiguous() or kc.shape != vc.shape or kc.shape[3] != hd or \
                    not (n1.is_cuda and n2.is_cuda and kc.is_cuda and vc.is_cuda):
                return None
            e = k = 0
            if lw.router is not None:
                moe, r = cfg.ff_type.moe, lw.router
                e, k = moe.num_experts, moe.num_experts_per_token
                up, down, bias = lw.experts_gate_up, lw.experts_down, lw.expert_bias
                if lw.shared_gate_up is not None or lw.expert_base or up.experts != e or r.dtype != bf16 or not r.is_contiguous() or \
                        not r.is_cuda or (bias is not None and (not bias.is_cuda or bias.dtype != torch.float32 or not bias.is_contiguous())):
                    return None
                pairs, most = max(pairs, t * k), max(most, e)
                if narrow.pays_grouped(up, down, t * k):
                    r_up = r_down = self.NARROW
                    if t <= ROUTER_ROWS and r.data_ptr() % 16 == 0:
                        r_up |= self.WITH_NORM
                    y = max(y, t * k * d * 4)
                else:
                    up, down = grouped._expanded_if_needed(up), grouped._expanded_if_needed(down)
                    if not (grouped._grouped_ok(up) and grouped._grouped_ok(down) and up.w.is_contiguous() and down.w.is_contiguous()):
                        return None
                    r_up, r_down = self._tiles(up, t * k, e, True), self._tiles(down, t * k, e)
                    xs, y = max(xs, t * k * d * 2), max(y, t * k * d * 2)
                act = max(act, t * k * up.n)
            else:
                up, down = lw.w_gate_up, lw.w_down
                r_up, r_down = self._gate_up(up, t, n2), self._plain(down, t)
                act, mid = max(act, t * up.n), max(mid, 0 if r_up & self.SWIGLU else t * up.n * 2)
            r_qkv, r_out = self._normed(lw.wqkv, t, n1), self._plain(lw.wo, t)
            if not (r_qkv and r_out and r_up and r_down):
                return None
            recs.extend((p1, p2, kc.data_ptr(), vc.data_ptr(), cache.k_sb[li].data_ptr() if q8 else 0,
                         cache.v_sb[li].data_ptr() if q8 else 0, 0 if not e else lw.router.data_ptr(),
                         0 if not e or bias is None else bias.data_ptr(), e, k))
            for w, route in ((lw.wqkv, r_qkv), (lw.wo, r_out), (up, r_up), (down, r_down)):
                s, b = w.scales, w.biases
                if not w.w.is_cuda or (s is not None and not (s.is_cuda and b.is_cuda)):
                    return None
                # a weight of the weight-streaming kernel has been looked at for it (narrow.supported)
                if route & 15 != self.NARROW and s is not None and not (s.is_contiguous() and b.is_contiguous() and w.w.is_contiguous()):
                    return None
                if route & 15 == self.EXPAND:
                    dense = max(dense, w.n * w.k * 2)
                recs.extend((w.w.data_ptr(), 0 if s is None else s.data_ptr(), 0 if b is None else b.data_ptr(), w.n, w.k,
                             w.experts if e else 0, w.kind, int(s is not None and w.scales_f16), route))
        few = few_rows_plan(t, hq, hkv, hd, pos0 + t, q8)
        kv_bytes = pages * hkv * 16 * hd * 2 if q8 and not few else 0
        rows, heads, routes = t * d * 2, t * hq * hd * 2, pairs * 4
        offsets, size = prompt_offsets((                   # prefill_plan.PIECES
            rows, rows, rows, t * (hq + 2 * hkv) * hd * 2, heads, heads, act, mid, dense, kv_bytes, kv_bytes, t * most * 4, routes, routes, most * 4,
            (most + 1) * 4 if most else 0, routes, most * 4, routes, xs, y))
        ws = torch.empty(size, dtype=torch.uint8, device=m.device)
        base = ws.data_ptr()
        iota, zeros = self._tables(pos0 + t + 1)
        window = int(cfg.sliding_window or 0)
        head = array.array("q", (
            len(mw.layers), t, d, hq, hkv, hd, pos0, window, row.numel(), 16, cache.k[0].shape[0], int(cfg.rope_traditional),
            int(not few and prefill_kernel_choice(hd, window) == "tc"), int(os.environ.get("RMLX_FLASH_PREFILL_LANES", "0")), pages, few, mw.embed.shape[0],
            mw.embed.data_ptr(), token_ids.data_ptr(), row.data_ptr(), iota.data_ptr() + 4 * pos0, zeros.data_ptr(), iota.data_ptr(),
            m.cos.data_ptr(), m.sin.data_ptr(), GemmStatus.get(m.device).data_ptr(), *[base + o for o in offsets]))
        lib = _lib.cuda()
        if not self._words:
            words = (ctypes.c_int * 2)()
            lib.rmlx_prompt_sizes(words)
            self._words = tuple(words)
        assert self._words == (len(head), len(recs) // len(mw.layers)), "the records of csrc/runtime/prompt_run.cu"
        launches, what = ctypes.c_int(0), ctypes.c_char_p()
        rc = lib.rmlx_prompt_run(head.buffer_info()[0], recs.buffer_info()[0], cfg.rms_norm_eps, m.scale, ctypes.byref(launches),
                                 ctypes.byref(what), _lib.stream_ptr())
        _lib.count_launches(launches.value - 1)
        _lib.check(rc, (what.value or b"prompt_run").decode())
        return ws[:t * d * 2].view(bf16).view(t, d)


class NativePrefill:
    """Callable ``(token_ids, cache, seq_id) -> last-token logits [1, vocab]`` (fp32); with
    ``all_logits=True`` the logits of every position of the call, ``[T, vocab]`` (what speculative
    verification needs: crates/rmlx-nn/src/sampler.rs verify helpers read one row per proposal)."""

    def __init__(self, model, chunk: int = 8192):
        self.m = model
        self.chunk = chunk
        self.layers = _Layers(model)
        self.at_once = PromptRun(model)

    @torch.no_grad()
    def __call__(self, token_ids: torch.Tensor, cache: PagedKvCache, seq_id: int,
                 all_logits: bool = False) -> torch.Tensor:
        parts = []
        for s in range(0, token_ids.numel(), self.chunk):
            parts.append(self._chunk(token_ids[s:s + self.chunk], cache, seq_id, all_logits))
        return torch.cat(parts, 0) if all_logits else parts[-1]

    def _chunk(self, token_ids, cache, seq_id, all_logits=False):
        m = self.m
        cfg = m.cfg
        t = token_ids.numel()
        hd, hq, hkv = cfg.head_dim, m.hq, m.hkv
        pos0 = cache.seq_len(seq_id)
        cache.reserve(seq_id, t)
        token_ids = token_ids.to(torch.int32)
        h = self.at_once.run(token_ids, cache, seq_id, pos0)
        if h is not None:
            cache.commit(seq_id, t)
            GemmStatus.check(m.device)
            return self.layers.logits(h if all_logits else h[t - 1:t])
        row = cache.block_table[cache.slot_of[seq_id]]
        pos = torch.arange(pos0, pos0 + t, dtype=torch.int32, device=m.device)
        seq = torch.zeros(t, dtype=torch.int32, device=m.device)
        q = torch.empty(t, hq, hd, dtype=torch.bfloat16, device=m.device)

        npages = (pos0 + t + cache.block_size - 1) // cache.block_size
        ident = torch.arange(npages, dtype=torch.int32, device=m.device) if cache.quantized else None
        few = few_rows_plan(t, hq, hkv, hd, pos0 + t, cache.quantized)
        lens = pos + 1 if few else None

        def attend(li, qkv):
            D.rope_kv_write(qkv, q, cache.k[li], cache.v[li], row.view(1, -1), pos, m.cos, m.sin,
                            hq, hkv, token_seq=seq, traditional=cfg.rope_traditional, **cache.sb(li))
            if few:
                return few_rows_attention(q, cache.k[li], cache.v[li], row, lens, few, m.scale, cfg.sliding_window or 0, **cache.sb(li))
            if cache.quantized:
                # prompt attention over an 8-bit cache: the sequence's pages are expanded once per
                # layer into contiguous bf16 pages (amortised over the chunk's tokens)
                kk = D.kv_dequant_pages(cache.k[li], cache.k_sb[li], row, npages)
                vv = D.kv_dequant_pages(cache.v[li], cache.v_sb[li], row, npages)
                return flash_prefill_paged(q, kk, vv, ident, pos0, m.scale, cfg.sliding_window or 0)
            return flash_prefill_paged(q, cache.k[li], cache.v[li], row, pos0, m.scale,
                                       cfg.sliding_window or 0)

        h = self.layers.run(D.embedding(m.w.embed, token_ids), attend)
        cache.commit(seq_id, t)
        GemmStatus.check(m.device)
        return self.layers.logits(h if all_logits else h[t - 1:t])


class BatchedDecode:
    """One decode step for up to ``max_batch`` sequences through the tensor-core kernels; shapes are
    static (idle rows point at the reserved page 0), so the step is one CUDA graph."""

    def __init__(self, model, cache: PagedKvCache, max_batch: int, use_graph: bool = True,
                 splits: Optional[int] = None):
        self.m, self.cache, self.B = model, cache, max_batch
        self.layers = _Layers(model)
        cfg, dev = model.cfg, model.device
        b = max_batch
        self.tokens = torch.zeros(b, dtype=torch.int32, device=dev)
        self.positions = torch.zeros(b, dtype=torch.int32, device=dev)
        self.seq_lens = torch.zeros(b, dtype=torch.int32, device=dev)
        self.rows = torch.arange(b, dtype=torch.int32, device=dev)
        self.live = torch.zeros(b, dtype=torch.int32, device=dev)
        self.table = torch.zeros(b, cache.max_blocks_per_seq, dtype=torch.int32, device=dev)
        self.q = torch.empty(b, model.hq, cfg.head_dim, dtype=torch.bfloat16, device=dev)
        self.next_tokens = torch.zeros(b, dtype=torch.int32, device=dev)
        # one captured graph per batch bucket: a step runs the smallest bucket that holds the
        # bound rows (crates/rmlx-metal/src/icb.rs:357, a replay cache keyed by shape)
        self.buckets = tuple(x for x in (1, 2, 4, 8, 16, 32, 64) if x < b) + (b,)
        self.graphs = GraphCache(max_entries=len(self.buckets))
        self._splits_arg = splits
        self._fd = {}
        self.splits, self.fd = self._fd_plan(b)
        self.argmax_scratch = D.ArgmaxScratch(b, dev)
        self.seq_ids: List[int] = []
        self.launches_per_step = 0           # launches of this package's kernels in one step
        self.use_graph = use_graph and model.layout.world == 1 and not _lib.debug_serialize()
        self._logits = {}
        self._last_bucket = b

    def _fd_plan(self, nb: int):
        if nb not in self._fd:
            m, cfg = self.m, self.m.cfg
            sp = self._splits_arg or D.default_splits(
                nb, m.hkv, _lib.cuda().rmlx_flash_decode_gtiles(m.hq, m.hkv),
                self.cache.max_blocks_per_seq * 16)
            self._fd[nb] = (sp, D.FlashDecodeScratch(nb, m.hq, m.hkv, cfg.head_dim, sp, m.device, max_len=None if self._splits_arg
                                                     else self.cache.max_blocks_per_seq * 16))
        return self._fd[nb]

    def bucket(self) -> int:
        return bucket_for(max(1, len(self.seq_ids)), self.buckets)

    def bind(self, seq_ids: Sequence[int], last_tokens: Sequence[int]) -> None:
        assert len(seq_ids) <= self.B
        self.seq_ids = list(seq_ids)
        n = len(seq_ids)
        lens = [self.cache.seq_len(s) for s in seq_ids]
        # idle rows attend to one (zero) key on the reserved page 0 and never advance
        self.tokens.zero_(); self.positions.zero_(); self.seq_lens.fill_(1); self.live.zero_()
        self.tokens[:n] = torch.tensor(list(last_tokens), dtype=torch.int32)
        self.positions[:n] = torch.tensor(lens, dtype=torch.int32)
        self.seq_lens[:n] = torch.tensor([l + 1 for l in lens], dtype=torch.int32)
        self.live[:n] = 1
        self._saved_tokens = self.tokens.clone()
        self.refresh_tables()

    def refresh_tables(self) -> None:
        self.table.zero_()
        for i, s in enumerate(self.seq_ids):
            self.table[i].copy_(self.cache.block_table[self.cache.slot_of[s]])

    def reserve(self, steps: int) -> None:
        for s in self.seq_ids:
            self.cache.reserve(s, steps)
        self.refresh_tables()

    def _body(self, nb: Optional[int] = None) -> None:
        m, cfg, cache = self.m, self.m.cfg, self.cache
        nb = self.B if nb is None else nb
        splits, fd = self._fd_plan(nb)
        tokens, positions, seq_lens = self.tokens[:nb], self.positions[:nb], self.seq_lens[:nb]
        table, q, rows, live = self.table[:nb], self.q[:nb], self.rows[:nb], self.live[:nb]

        def attend(li, qkv):
            D.rope_kv_write(qkv, q, cache.k[li], cache.v[li], table, positions, m.cos,
                            m.sin, m.hq, m.hkv, token_seq=rows, traditional=cfg.rope_traditional,
                            **cache.sb(li))
            return D.flash_decode_paged(q, cache.k[li], cache.v[li], table, seq_lens,
                                        m.scale, splits, fd, cfg.sliding_window or 0, **cache.sb(li))

        h = self.layers.run(D.embedding(m.w.embed, tokens), attend)
        self._logits[nb] = self.layers.logits(h)
        D.argmax(self._logits[nb], self.next_tokens[:nb], self.argmax_scratch)
        # feed the tokens back and advance the bound rows (idle rows stay at length 0 on page 0)
        tokens.copy_(self.next_tokens[:nb] * live)
        positions.add_(live)
        seq_lens.add_(live)

    @property
    def logits(self) -> Optional[torch.Tensor]:
        """Logits of the last step: [bucket rows, vocab] (rows beyond the bound sequences are idle)."""
        return self._logits.get(self._last_bucket)

    @torch.no_grad()
    def step(self) -> torch.Tensor:
        """Run one step for every bound sequence; returns the next-token ids (device, int32)."""
        nb = self._last_bucket = self.bucket()
        if not self.use_graph:
            n0 = _lib.launch_count()
            self._body(nb)
            self.launches_per_step = _lib.launch_count() - n0
        else:
            def body():
                n0 = _lib.launch_count()
                self._body(nb)
                self.launches_per_step = _lib.launch_count() - n0
            # one warm-up run outside capture (lazy initialisations), state rewound after each
            self.graphs.get_or_capture(("batched", nb), body, warmup=1, restore=self._rewind,
                                       device=self.m.device).replay()
        for s in self.seq_ids:
            self.cache.commit(s, 1)
        return self.next_tokens

    def set_next_tokens(self, tokens: Sequence[int]) -> None:
        """Replace the tokens the last step fed back (its arg-max) with ones chosen by the caller,
        e.g. sampled from ``logits``; positions and lengths were already advanced by the step."""
        n = len(self.seq_ids)
        assert len(tokens) == n
        self.tokens[:n] = torch.tensor([int(t) for t in tokens], dtype=torch.int32)
        self._saved_tokens = self.tokens.clone()

    def _rewind(self) -> None:
        """Undo the state advance of a warm-up step (the KV slot it wrote is rewritten by the real one)."""
        n = len(self.seq_ids)
        lens = [self.cache.seq_len(s) for s in self.seq_ids]
        self.positions.zero_(); self.seq_lens.fill_(1)
        self.positions[:n] = torch.tensor(lens, dtype=torch.int32)
        self.seq_lens[:n] = torch.tensor([l + 1 for l in lens], dtype=torch.int32)
        self.tokens.copy_(self._saved_tokens)

    @torch.no_grad()
    def generate(self, steps: int) -> torch.Tensor:
        self.reserve(steps + 1)
        self._saved_tokens = self.tokens.clone()
        out = torch.zeros(len(self.seq_ids), steps, dtype=torch.int64)
        for i in range(steps):
            nxt = self.step()
            out[:, i] = nxt[:len(self.seq_ids)].cpu().long()
            self._saved_tokens = self.tokens.clone()
        GemmStatus.check(self.m.device)
        return out


def plan_chunk(model, scratch_limit_bytes: int = 4 << 30, longest: int = 8192) -> int:
    """Largest prompt chunk (a multiple of 128, at most ``longest``) whose per-layer intermediates
    stay within ``scratch_limit_bytes`` according to the layer's static plan
    (``models.prefill_plan.PrefillPlan``, which lays them out as the portion itself does). Not counted, because no chunk makes
    them fewer: an 8-bit cache's pages, expanded for the whole context, one layer at a time."""
    kinds = [w for l in getattr(getattr(model, "w", None), "layers", ()) for w in (l.wqkv, l.wo, l.w_gate_up, l.w_down) if w is not None]
    weights = "q8" if any(w.kind == W_Q8 or (w.kind == W_Q4 and w.scales_f16) for w in kinds) else \
        "q4" if any(w.kind == W_Q4 for w in kinds) else "bf16"
    chunk = longest
    while chunk > 128 and PrefillPlan(model.cfg, chunk, model.layout, weights).scratch_bytes > scratch_limit_bytes:
        chunk -= 128
    return chunk


def enable_native_prefill(model, chunk: Optional[int] = None, scratch_limit_bytes: int = 4 << 30) -> bool:
    """Attach the native path to ``model.prefill``; False (and the library-kernel path stays) when the
    model's shapes are outside what the kernels cover. ``chunk`` None: the longest chunk whose
    intermediates fit ``scratch_limit_bytes`` (``plan_chunk``)."""
    try:
        if chunk is None:
            chunk = plan_chunk(model, scratch_limit_bytes)
        model._native_prefill = NativePrefill(model, chunk)
        return True
    except ImportError:
        return False
