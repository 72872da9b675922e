"""Static plans and scratch for prompt processing.

``PrefillPlan`` lists, for a sequence length, the launches of one layer with their shapes and the
scratch each needs (the reference builds the same per-length ``PlanStep`` lists,
crates/rmlx-nn/src/prefill_plan.rs:16-300); ``prompt_offsets`` lays that scratch out in one block, for the plan and for
the portion that runs alike; ``PrefillPool`` keeps a few slots of pre-allocated
intermediates sized for the largest planned length so that chunks of a prompt do not allocate
(crates/rmlx-nn/src/prefill_pool.rs:33-160, crates/rmlx-nn/src/dynamic.rs:16-104).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Dict, List, Optional, Sequence, Tuple

import torch

from ..config import TransformerConfig
from .weights import ParallelLayout


@dataclass(frozen=True)
class PlanStep:
    name: str
    kernel: str
    m: int
    n: int
    k: int
    out_bytes: int

    @property
    def flops(self) -> float:
        return 2.0 * self.m * self.n * self.k


#: The pieces of a portion's work space, in the order of the native call's record (csrc/runtime/prompt_run.cu).
PIECES = ("h0", "h1", "xn", "qkv", "q", "attn", "act", "mid", "dense", "kk", "vv", "logits", "idx", "wts", "counts", "offsets", "order",
          "cursors", "row_of", "xs", "y")


def prompt_offsets(sizes: Sequence[int]) -> Tuple[List[int], int]:
    """Where the pieces of a portion's work space lie in one block (bytes from its start, 256-byte addresses, in the order of ``PIECES``), and
    the block's size. ``sizes``: bytes of each piece. A launch writes only after the one before it has finished, so what no later
    launch reads is free.

    The residual stream, a weight expanded for one product and the routing's tables have places of their own. The rest belongs to one
    half of a layer and is dead in the other, so the halves share their memory; and within a half a piece lies where one was
    that has been read by then (queries on the normed rows, the heads' results on qkv, ...). Written out: a portion of a few rows waits for
    this (3 us, 8 by names)."""
    h0, h1, xn, qkv, q, attn, act, mid, dense, kk, vv, logits, idx, wts, counts, offsets, order, cursors, row_of, xs, y = \
        [s + 255 & ~255 for s in sizes]
    at_dense = h0 + h1
    at_idx = at_dense + dense
    at_wts = at_idx + idx
    at_counts = at_wts + wts
    at_offsets = at_counts + counts
    at_order = at_offsets + offsets
    at_cursors = at_order + order
    at_row_of = at_cursors + cursors
    shared = at_row_of + row_of
    # attention: normed rows, then queries; qkv, then the heads' results; expanded pages
    at_qkv = shared + (xn if xn > q else q)
    at_kk = at_qkv + (qkv if qkv > attn else attn)
    at_vv = at_kk + kk
    # feed-forward: normed rows; logits, then the gated rows; both halves of the gate, sorted rows or the experts' results
    at_act = shared + xn
    at_mid = at_act + (logits if logits > act else act)
    return [0, h0, shared, at_qkv, shared, at_qkv, at_act, at_mid, at_dense, at_kk, at_vv, at_act, at_idx, at_wts, at_counts, at_offsets, at_order,
            at_cursors, at_row_of, at_mid, at_mid], max(at_vv + vv, at_mid + max(mid, xs, y))


def prompt_block(sizes: Dict[str, int]) -> Tuple[Dict[str, int], int]:
    """``prompt_offsets`` by name; pieces that are left out are empty."""
    at, total = prompt_offsets([sizes.get(name, 0) for name in PIECES])
    return dict(zip(PIECES, at)), total


class PrefillPlan:
    """The launches of one layer for ``seq_len`` tokens, and their scratch. ``weights``: "bf16", "q4" or "q8", as the projections are
    stored; with ``kv_quant`` ("q8") the pages of ``context`` tokens (the portion's own if that is more) are expanded beside them."""

    def __init__(self, cfg: TransformerConfig, seq_len: int, layout: Optional[ParallelLayout] = None, weights: str = "bf16",
                 kv_quant: Optional[str] = None, context: int = 0):
        layout = layout or ParallelLayout()
        hq, _, hkv, _ = layout.heads(cfg)
        d, hd, t = cfg.hidden_size, cfg.head_dim, seq_len
        self.cfg, self.seq_len = cfg, seq_len
        steps: List[PlanStep] = [
            PlanStep("attn_norm", "rms_norm", t, d, 1, t * d * 2),
            PlanStep("qkv", "gemm", t, (hq + 2 * hkv) * hd, d, t * (hq + 2 * hkv) * hd * 2),
            PlanStep("rope_kv", "rope_kv_write", t, (hq + 2 * hkv) * hd, 1, t * hq * hd * 2),
            PlanStep("attention", "flash_prefill", t, hq * hd, t // 2 + 1, t * hq * hd * 2),
            PlanStep("o_proj", "gemm+residual", t, d, hq * hd, t * d * 2),
            PlanStep("ffn_norm", "rms_norm", t, d, 1, t * d * 2),
        ]
        if cfg.ff_type.kind == "moe":
            m = cfg.ff_type.moe
            k, inter = m.num_experts_per_token, m.intermediate_dim // layout.world
            steps += [
                PlanStep("router", "gemm_f32+topk", t, m.num_experts, d, t * k * 8),
                PlanStep("scatter", "moe_scatter_rows", t * k, d, 1, t * k * d * 2),
                PlanStep("gate_up", "grouped_gemm+swiglu", t * k, 2 * inter, d, t * k * inter * 2),
                PlanStep("down", "grouped_gemm", t * k, d, inter, t * k * d * 2),
                PlanStep("combine", "moe_combine+residual", t, d, k, t * d * 2),
            ]
        else:
            inter = cfg.ff_type.intermediate_dim // layout.world
            steps += [
                PlanStep("gate_up", "gemm+swiglu", t, 2 * inter, d, t * inter * 2),
                PlanStep("down", "gemm+residual", t, d, inter, t * d * 2),
            ]
        self.steps: Tuple[PlanStep, ...] = tuple(steps)
        # one block holds it all (models/prefill.py: PromptRun); tensor parallelism and shared experts allocate launch by launch
        moe = cfg.ff_type.moe if cfg.ff_type.kind == "moe" else None
        self.at_once = layout.world == 1 and not (moe is not None and moe.num_shared_experts)

        def expands(k: int) -> bool:       # products of more than a few rows: 8-bit weights, and 4-bit ones outside the kernels' groups
            return weights == "q8" or (weights == "q4" and k % 512 != 0)

        pages = -(-max(t, context) // 16) * hkv * 16 * hd * 2 if kv_quant else 0
        p = self.pieces = dict(h0=t * d * 2, h1=t * d * 2, xn=t * d * 2, qkv=t * (hq + 2 * hkv) * hd * 2, q=t * hq * hd * 2,
                               attn=t * hq * hd * 2, kk=pages, vv=pages, act=0, mid=0)
        linear = [((hq + 2 * hkv) * hd, d), (d, hq * hd)]
        dense = [inter] if moe is None else \
            [cfg.dense_intermediate_dim // layout.world] if cfg.first_dense_layers and cfg.dense_intermediate_dim else []
        for i in dense:
            linear += [(2 * i, d), (d, i)]
            p["act"] = t * i * 2
            p["mid"] = t * 2 * i * 2 if expands(d) or 2 * i % 256 else 0
        p["dense"] = max([n * k * 2 for n, k in linear if expands(k)], default=0)
        if moe is not None:
            pairs, e = t * moe.num_experts_per_token, moe.num_experts
            p["act"] = max(p["act"], pairs * inter * 2)
            p.update(logits=t * e * 4, idx=pairs * 4, wts=pairs * 4, counts=e * 4, offsets=(e + 1) * 4, order=pairs * 4, cursors=e * 4,
                     row_of=pairs * 4, xs=pairs * d * 2)
            # few pairs of quantised experts are added up in fp32, without sorted rows
            p["y"] = pairs * d * (4 if weights != "bf16" and pairs <= 16 * e else 2)

    @property
    def scratch_bytes(self) -> int:
        """Bytes beside weights and cache: the block of the native call; launch by launch, all intermediates of a layer (each lives until
        its name is used again)."""
        return prompt_block(self.pieces)[1] if self.at_once else sum(self.pieces.values())

    @property
    def flops(self) -> float:
        return sum(s.flops for s in self.steps if "gemm" in s.kernel or s.kernel == "flash_prefill")


class PrefillPool:
    """``slots`` scratch buffers of ``bytes_per_slot`` each; ``acquire`` hands out a free one (or
    None when all are in use), ``release`` returns it."""

    def __init__(self, bytes_per_slot: int, slots: int = 4, device="cpu"):
        self.bytes_per_slot = int(bytes_per_slot)
        self._bufs = [torch.empty(self.bytes_per_slot, dtype=torch.uint8, device=device) for _ in range(slots)]
        self._free = list(range(slots))
        self._plans: Dict[int, PrefillPlan] = {}

    @classmethod
    def for_config(cls, cfg: TransformerConfig, max_seq_len: int, slots: int = 4, device="cpu",
                   layout: Optional[ParallelLayout] = None) -> "PrefillPool":
        pool = cls(PrefillPlan(cfg, max_seq_len, layout).scratch_bytes, slots, device)
        pool._cfg, pool._layout = cfg, layout
        return pool

    def plan(self, seq_len: int) -> PrefillPlan:
        p = self._plans.get(seq_len)
        if p is None:
            p = PrefillPlan(self._cfg, seq_len, self._layout)
            if p.scratch_bytes > self.bytes_per_slot:
                raise ValueError("sequence longer than the pool was sized for")
            self._plans[seq_len] = p
        return p

    def acquire(self) -> Optional[Tuple[int, torch.Tensor]]:
        if not self._free:
            return None
        i = self._free.pop()
        return i, self._bufs[i]

    def release(self, slot: int) -> None:
        if slot in self._free or not 0 <= slot < len(self._bufs):
            raise ValueError("slot is not in use")
        self._free.append(slot)

    @property
    def available(self) -> int:
        return len(self._free)


class DynamicExecContext:
    """``count`` intermediates of [max_seq_len, hidden] allocated once; a step of any length up to
    the maximum takes views of their first rows, so a varying sequence length never allocates
    (crates/rmlx-nn/src/dynamic.rs:16-104)."""

    def __init__(self, max_seq_len: int, hidden_dim: int, dtype=torch.bfloat16, num_intermediates: int = 4,
                 device="cpu"):
        if max_seq_len < 1 or hidden_dim < 1 or num_intermediates < 1:
            raise ValueError("DynamicExecContext: sizes must be positive")
        self._max, self._hidden, self.dtype = max_seq_len, hidden_dim, dtype
        self._bufs = [torch.zeros(max_seq_len, hidden_dim, dtype=dtype, device=device)
                      for _ in range(num_intermediates)]

    def max_seq_len(self) -> int:
        return self._max

    def hidden_dim(self) -> int:
        return self._hidden

    def num_intermediates(self) -> int:
        return len(self._bufs)

    def allocated_bytes(self) -> int:
        return sum(b.numel() * b.element_size() for b in self._bufs)

    def get_intermediate(self, idx: int, actual_seq_len: int) -> torch.Tensor:
        """A view of the first ``actual_seq_len`` rows of intermediate ``idx`` (no copy)."""
        if not 0 <= idx < len(self._bufs):
            raise ValueError(f"DynamicExecContext: intermediate index {idx} >= count {len(self._bufs)}")
        if not 0 <= actual_seq_len <= self._max:
            raise ValueError(f"DynamicExecContext: actual_seq_len {actual_seq_len} > max_seq_len {self._max}")
        return self._bufs[idx][:actual_seq_len]
