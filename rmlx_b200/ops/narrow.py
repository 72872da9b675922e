"""Projections of a few rows on csrc/kernels/narrow_gemm.cu: decode batches, short prompts and verification. The weights
(bf16, 4-bit or 8-bit) are streamed once through registers, eight rows of x per tensor-core instruction; the grouped form
takes (row, slot) pairs by expert. Counterpart of the reference's small-M qmm / gather_qmm kernels
(crates/rmlx-core/src/ops/quantized.rs:2755,9634)."""
from __future__ import annotations

from typing import Optional

import torch

from .. import _lib
from .weights import LinearWeight, W_BF16, W_Q4, W_Q8

_lib.register_cuda_sigs({
    "rmlx_narrow_supported": ("iii", "i"),
    "rmlx_narrow_gemm": ("ippppiippipfpipiiiiiiiiip", "i"),
    "rmlx_narrow_pairs": ("ippppiipipfpiiiiiiip", "i"),
    "rmlx_narrow_group": ("piippip", "i"),
    "rmlx_narrow_combine": ("ppippipiiiiip", "i"),
})


def supported(w: LinearWeight) -> bool:
    """Whether the kernel takes this weight (``rmlx_narrow_supported``, in Python because it is asked before every projection):
    whole 16-row tiles, K a multiple of 512 (bf16 weights: 64), up to 256 experts, and every table contiguous and at a 16-byte
    address, as the copies of 16 bytes need it (views that are not keep the kernels that take them)."""
    t, s, b = w.w, w.scales, w.biases
    shape = t.shape
    if shape[-2] % 16 or (len(shape) == 3 and shape[0] > 256) or not t.is_contiguous():
        return False
    if w.kind == W_BF16:
        return t.dtype == torch.bfloat16 and shape[-1] % 64 == 0 and shape[-1] > 0 and t.data_ptr() % 16 == 0
    return (t.dtype == torch.int32 and shape[-1] % (64 if w.kind == W_Q4 else 128) == 0 and shape[-1] > 0 and s is not None and
            b is not None and s.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and s.is_contiguous() and
            b.is_contiguous() and (t.data_ptr() | s.data_ptr() | b.data_ptr()) % 16 == 0)


def pays(w: LinearWeight, rows: int) -> bool:
    """Whether a plain projection of ``rows`` rows is faster here than on the 128-row tensor-core tiles (and takes this weight).

    Measured (us, this kernel / the tiles of 128 rows of x). 4-bit: 28672 x 4096 25 / 39 at 16 rows, 43 / 39 at 24; 28672 x 8192 44 / 72 at 16, 75 /
    72 at 24; 9216 x 4096 15 / 26 at 16; 4096 x 8192 20 / 45 at 32; 4096 x 14336 37 / 74: up to 16 rows, and up to 32 for moderate widths, except
    where the tiles are one round of the SMs and K is short: at 17 to 24 rows 8192 x 512 9 / 8, 8192 x 1024 12 / 11, 6144 x 1024 7 / 10, 8192 x 2048
    15 / 19; at 32 rows, two passes of two tiles, 6144 x 512 11 / 7, 8192 x 2048 19 / 15, 8192 x 2560 23 / 18, 8192 x 4096 25 / 25; 12288 wide
    512 12 / 10, 1024 14 / 16. 8-bit weights would be expanded first: up to 32 rows; above, short small ones take longer here (at 64 rows 2048 x
    1024 14 / 9, 2048 x 3072 21 / 19, 4096 x 2048 20 / 19, 4096 x 2560 25 / 22, 8192 x 512 13 / 12; 16384 x 2048 33 / 50, 28672 x 4096
    99 / 165). bf16, 9216 x 4096: 20 / 28 at 16 rows; 28672 x 4096: 46 / 45:
    eight rows, and 16 for up to 16384 rows of W; large weights stream at the copy bandwidth on the tiles too (at 5 rows
    28672 x 8192 89 / 119, 65536 x 4096 101 / 103, 151936 x 4096 227 / 214; at 8 rows 32768 x 4096 53 / 72, 28672 x 8192 89 / 84,
    65536 x 4096 101 / 100). Weights of less than a million entries take a tile's time anyway."""
    n, k = w.n, w.k
    entries = n * k
    if rows < 1 or rows > 64 or entries < 1 << 20:
        return False
    if w.kind == W_BF16:
        ok = (rows <= 8 and entries <= (1 << 27 if rows > 5 else 1 << 28)) or (rows <= 16 and n <= 16384)
    elif w.kind == W_Q4:
        ok = rows <= 16 or (rows <= 32 and n <= 12288 and (
            n <= 4096 or (rows <= 24 and (n <= 6144 or n > 9472 or k >= 1536)) or k >= (1024 if n > 9472 else 3072)))
    else:
        ok = rows <= 32 or k >= 4096 or entries >= 12 << 20 or (n >= 6144 and k >= 1024)
    return ok and supported(w)


def pays_grouped(gate_up: LinearWeight, down: LinearWeight, pairs: int) -> bool:
    """Whether an expert feed-forward of ``pairs`` (row, slot) pairs is faster here: up to twelve pairs per expert in 4 bits, fourteen in 8
    (128 experts of 4096 x 1536, both projections, us, here / on the tiles: 4-bit 382 / 470 at 1024 pairs, 466 / 480 at 1600, 577 / 490 at
    2048; 8-bit on expanded weights 586 / 815 at 1024, 748 / 894 at 2048; at 14 and 16 pairs per expert 32 of 2048 x 2048 0.89 and 1.06 of their
    time, 64 of 2048 x 1024 0.94 and 1.07), eight where the experts are few and small (16 of 1024 x 512 at 10: 4-bit 35 / 33, 8-bit 34 / 27). bf16
    experts are as fast on the tiles (523 + 275 against 549 + 305 at 512 pairs)."""
    most = 8 if gate_up.experts * gate_up.n * gate_up.k < 1 << 27 else 12 if gate_up.kind == W_Q4 else 14
    return (gate_up.kind in (W_Q4, W_Q8) and down.kind == gate_up.kind and 0 < pairs <= most * gate_up.experts and
            gate_up.n * gate_up.k >= 1 << 20 and supported(gate_up) and supported(down))


def _holds(t: torch.Tensor, rows: int, columns: int) -> bool:
    """At least so many rows and columns, columns side by side."""
    shape = t.shape
    return len(shape) == 2 and shape[0] >= rows and shape[1] >= columns and t.stride(1) == 1


def same_layout(residual: torch.Tensor, out: Optional[torch.Tensor], rows: int, columns: int) -> bool:
    """Whether a residual is laid out as the result is (a new one without ``out``), which the tensor-core GEMMs ask for."""
    return residual.shape == (rows, columns) and residual.stride() == ((columns, 1) if out is None else out.stride())


def narrow_gemm(x: torch.Tensor, w: LinearWeight, norm_w: Optional[torch.Tensor] = None, eps: float = 1e-6,
                residual: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None, out_dtype=torch.bfloat16,
                swiglu: bool = False, offsets: Optional[torch.Tensor] = None, order: Optional[torch.Tensor] = None,
                x_div: int = 1, rows: Optional[int] = None, tiles: int = 0, shares: int = 0, pdl: bool = False) -> torch.Tensor:
    """out = residual + rmsnorm(x; norm_w) W^T, or silu(gate) * up of a stacked [gate; up] weight with ``swiglu``.

    Grouped: w is [E, N, K], ``offsets`` int32 [E + 1] the positions of every expert's rows, ``order`` the output row of each
    position (None: the position itself), whose input is row ``output row // x_div`` of x; ``rows``: positions in all.
    ``tiles`` (eight rows of x each per pass: 1, 2, 4) and ``shares`` (of K) are chosen from the sizes when 0."""
    _lib.require_cuda_tensor(x, w.w)
    n_all, k = w.n, w.k
    shape, stride = x.shape, x.stride()
    assert x.dtype == torch.bfloat16 and len(shape) == 2 and stride[1] == 1 and shape[1] == k
    m = shape[0] if rows is None else rows
    n = n_all // 2 if swiglu else n_all
    if out is None:
        out = torch.empty(m, n, dtype=out_dtype, device=x.device)
    else:
        assert _holds(out, m, n)
    assert out.dtype in (torch.bfloat16, torch.float32)
    assert residual is None or (residual.dtype == torch.bfloat16 and _holds(residual, m, n))
    scales, biases = w.scales, w.biases
    rc = _lib.cuda().rmlx_narrow_gemm(
        w.kind, w.w.data_ptr(), scales if scales is None else scales.data_ptr(), biases if biases is None else biases.data_ptr(),
        x.data_ptr(), stride[0], x_div, order if order is None else order.data_ptr(),
        offsets if offsets is None else offsets.data_ptr(), 1 if offsets is None else w.experts,
        norm_w if norm_w is None else norm_w.data_ptr(), eps, residual if residual is None else residual.data_ptr(),
        0 if residual is None else residual.stride(0), out.data_ptr(), out.stride(0), out.dtype == torch.float32, m, n_all, k,
        swiglu, tiles, shares, pdl, _lib.stream_ptr())
    _lib.check(rc, "narrow_gemm")
    return out


def group_pairs(idx: torch.Tensor, experts: int, offsets: Optional[torch.Tensor] = None, order: Optional[torch.Tensor] = None,
                pdl: bool = False):
    """Pairs (row * k + slot) by chosen expert: (offsets [E + 1], order [rows * k]), int32. Choices outside [0, experts) are in
    no list: offsets[E] counts the others."""
    n = idx.numel()
    if offsets is None:
        offsets = torch.empty(experts + 1, dtype=torch.int32, device=idx.device)
    if order is None:
        order = torch.empty(n, dtype=torch.int32, device=idx.device)
    _lib.check(_lib.cuda().rmlx_narrow_group(idx.data_ptr(), n, experts, offsets.data_ptr(), order.data_ptr(), int(pdl),
                                             _lib.stream_ptr()), "narrow_group")
    return offsets, order


def combine(y: torch.Tensor, idx: torch.Tensor, experts: int, wts: torch.Tensor, residual: Optional[torch.Tensor] = None,
            out: Optional[torch.Tensor] = None, pdl: bool = False) -> torch.Tensor:
    """out[t] = residual[t] + sum over the slots whose choice idx[t, slot] is an expert of wts[t, slot] * y[t k + slot], y fp32."""
    t, k = wts.shape
    d = y.shape[1]
    if out is None:
        out = torch.empty(t, d, dtype=torch.bfloat16, device=y.device)
    _lib.check(_lib.cuda().rmlx_narrow_combine(y.data_ptr(), idx.data_ptr(), experts, wts.data_ptr(), _lib.ptr(residual),
                                               0 if residual is None else residual.stride(0), out.data_ptr(), out.stride(0), t, k,
                                               d, int(pdl), _lib.stream_ptr()), "narrow_combine")
    return out


def pays_shared(gate_up: LinearWeight, rows: int, top_k: int) -> bool:
    """Whether a decode step of ``rows`` rows should read every chosen expert once for all rows (four launches) rather than once
    per (row, slot) pair on the streaming kernels (two). Measured on whole two-layer steps (us, here / there), 128 experts of
    4096 x 1536 and 32 of 2048 x 2048: 4-bit 371 / 386 at 2 rows of the larger, 251 / 243 at 5 of the smaller and 277 / 313 at 8;
    8-bit 470 / 544 and 183 / 182 at 2; bf16 691 / 582 at 2 rows of the larger, 732 / 731 at 3, 877 / 930 at 4: there only the
    sharing itself helps, as pairs already stream at the copy bandwidth."""
    if gate_up.kind == W_BF16:
        return rows >= 4
    return rows >= 2 and rows * top_k * gate_up.n * gate_up.k >= (200e6 if gate_up.kind == W_Q4 else 60e6)


class ExpertScratch:
    """Buffers of ``expert_ffn`` and ``pairs_ffn`` for up to ``rows`` rows, for callers whose launches may not allocate. Experts narrower
    than those it was made for use the first columns of ``act``."""

    def __init__(self, rows: int, top_k: int, gate_up: LinearWeight, down: LinearWeight):
        dev, pairs = gate_up.device, rows * top_k
        self.offsets = torch.empty(gate_up.experts + 1, dtype=torch.int32, device=dev)
        self.order = torch.empty(pairs, dtype=torch.int32, device=dev)
        self.act = torch.empty(pairs, gate_up.n // 2, dtype=torch.bfloat16, device=dev)
        self.y = torch.empty(pairs, down.n, dtype=torch.float32, device=dev)


def expert_ffn(x: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor, gate_up: LinearWeight, down: LinearWeight,
               norm_w: Optional[torch.Tensor] = None, eps: float = 1e-6, residual: Optional[torch.Tensor] = None,
               out: Optional[torch.Tensor] = None, scratch: Optional[ExpertScratch] = None, pdl: bool = False) -> torch.Tensor:
    """residual + sum over slots of wts * down_e(silu(gate_e xn) * up_e xn), e = idx[row, slot], xn = rmsnorm(x; norm_w):
    every expert's weights are read once for all rows that chose it. Slots whose choice is no expert add nothing."""
    t, k = idx.shape
    pairs = t * k
    s = scratch or ExpertScratch(t, k, gate_up, down)
    offsets, order = group_pairs(idx, gate_up.experts, s.offsets, s.order[:pairs], pdl=pdl)
    act = narrow_gemm(x, gate_up, norm_w, eps, out=s.act[:pairs, :gate_up.n // 2], swiglu=True, offsets=offsets, order=order, x_div=k,
                      rows=pairs, pdl=pdl)
    y = narrow_gemm(act, down, out=s.y[:pairs], offsets=offsets, order=order, rows=pairs, pdl=pdl)
    return combine(y, idx, gate_up.experts, wts, residual, out, pdl=pdl)


PAIRS = 32       # (row, slot) pairs that ``pairs_ffn`` takes


def pays_pairs(gate_up: LinearWeight, down: LinearWeight, rows: int, top_k: int) -> bool:
    """Whether so few rows' pairs should be multiplied one by one (``pairs_ffn``, three launches): quantised experts, hardly any of which is
    chosen twice (at random choices a quarter more pairs than experts at most), and enough of them that the even split of the work
    outweighs its launches. Measured, chained (us: pairs / ``expert_ffn`` / streaming kernels). 4-bit, 128 experts of 4096 x 1536, 8 of
    them: 37.5 / 51 / 37.2 for one row, 51 / 61 / 60 for two, 79 / 89 / 107 for four; 8 of 4096 x 14336, two of them: 54 / 58 / 69, 93 / 97 /
    122, three rows 124 / 117 / 175; 64 of 2048 x 1536, six of them: 24 / 33 / 20, 32 / 39 / 31, three rows 38 / 42 / 42. 8-bit, 128 of 2048
    x 1024, 8 of them: 27 / 38 / 23, 35 / 48 / 36, four rows 50 / 61 / 61; 8 of 4096 x 3584, two of them: 30 / 34 / 35. 32 small pairs
    in 4 bits stream faster (2048 x 1024 among 64 experts 42 / 46 / 40, among 128 42 / 54 / 40; 30 of them 41 / 45 / 43), and beyond 2^27
    entries that are read for a second time sharing wins (16 of 8192 x 4096, two of them, four rows 100 / 88 / 135, in 8 bits 145 / 134 / 217;
    three rows 80 / 78 / 107; one of them, eight rows 99 / 90 / 138)."""
    pairs, e = rows * top_k, gate_up.experts
    if gate_up.kind not in (W_Q4, W_Q8) or down.kind != gate_up.kind or not 0 < pairs <= PAIRS or e < 1:
        return False
    entries = gate_up.n * gate_up.k + down.n * down.k
    read = pairs * entries * (0.5625 if gate_up.kind == W_Q4 else 1.0625)
    distinct = e * (1.0 - (1.0 - min(1.0, top_k / e)) ** rows)
    least = 150e6 if gate_up.kind == W_Q4 and pairs > 30 else 90e6
    return (read >= least and pairs <= 1.25 * distinct and (pairs - distinct) * entries <= 1 << 27 and gate_up.k <= 32768 and
            down.k <= 32768 and gate_up.n % 32 == 0 and
            gate_up.scales.dtype == down.scales.dtype == torch.bfloat16 and supported(gate_up) and supported(down))


def pairs_gemm(x: torch.Tensor, w: LinearWeight, idx: torch.Tensor, x_div: int, out: torch.Tensor, norm_w: Optional[torch.Tensor] = None,
               eps: float = 1e-6, swiglu: bool = False, pdl: bool = False) -> torch.Tensor:
    """out[i] = rmsnorm(x[i // x_div]; norm_w) W_e^T, e = idx[i] of the flattened choices; rows whose choice is no expert stay as they are."""
    _lib.require_cuda_tensor(x, w.w, idx)
    n, k, pairs = w.n, w.k, idx.numel()
    assert x.dtype == torch.bfloat16 and x.stride(1) == 1 and x.shape[1] == k and idx.dtype == torch.int32 and idx.is_contiguous()
    assert _holds(out, pairs, n // 2 if swiglu else n) and x.shape[0] * x_div >= pairs
    rc = _lib.cuda().rmlx_narrow_pairs(w.kind, w.w.data_ptr(), w.scales.data_ptr(), w.biases.data_ptr(), x.data_ptr(), x.stride(0), x_div,
                                       idx.data_ptr(), w.experts, _lib.ptr(norm_w), eps, out.data_ptr(), out.stride(0),
                                       int(out.dtype == torch.float32), pairs, n, k, int(swiglu), int(pdl), _lib.stream_ptr())
    _lib.check(rc, "narrow_pairs")
    return out


def pairs_ffn(x: torch.Tensor, idx: torch.Tensor, wts: torch.Tensor, gate_up: LinearWeight, down: LinearWeight, norm_w: torch.Tensor,
              eps: float, residual: torch.Tensor, out: torch.Tensor, scratch: ExpertScratch, pdl: bool = False) -> torch.Tensor:
    """``expert_ffn`` of so few rows that hardly any share an expert: every pair by itself, without the lists."""
    k = idx.shape[1]
    pairs = idx.numel()
    act = pairs_gemm(x, gate_up, idx, k, scratch.act[:pairs, :gate_up.n // 2], norm_w, eps, swiglu=True, pdl=pdl)
    y = pairs_gemm(act, down, idx, 1, scratch.y[:pairs], pdl=pdl)
    return combine(y, idx, gate_up.experts, wts, residual, out, pdl=pdl)
