"""Quantised and grouped tensor-core matmuls (csrc/kernels/xgemm_tcgen05.cu).

``qmm``: y = x @ dequant(W)^T for MLX-affine Q4 weights, dequantised inside the tcgen05 main loop.
Shapes whose K is not a multiple of 512 (the scale arrays' rows then miss TMA's 16-byte stride
rule) take the two-step path: expand the weight once to bf16, then the bf16 tensor-core GEMM.
"""
from __future__ import annotations

from typing import Optional

import torch

from .. import _lib
from . import narrow
from .gemm import GemmStatus, gemm_bf16
from .weights import LinearWeight, W_Q4

_lib.register_cuda_sigs({
    "rmlx_qgemm_supported": ("i", "i"),
    "rmlx_xgemm": ("ipppppppiiiiiiiifpip", "i"),
    "rmlx_pair_gemm_supported": ("iiiiii", "i"),
    "rmlx_pair_gemm": ("ipppppppiiiiiiifpip", "i"),
    "rmlx_row_gemm_supported": ("iiiii", "i"),
    "rmlx_row_gemm": ("pppppippiiiiiiifipip", "i"),
    "rmlx_moe_scatter_rows": ("pipppppiiiip", "i"),
    "rmlx_moe_combine": ("ppppipiiiip", "i"),
})


def xgemm(x: torch.Tensor, w: LinearWeight, residual: Optional[torch.Tensor] = None,
          out: Optional[torch.Tensor] = None, offsets: Optional[torch.Tensor] = None, bn: int = 0,
          pdl: bool = False, swiglu: bool = False, gate_limit: float = 0.0) -> torch.Tensor:
    """Plain (offsets None) or grouped tensor-core GEMM with bf16 or Q4 weights.
    Grouped: x rows sorted by expert, ``offsets`` int32 [E+1] on the device, w stacked [E, N, K].
    ``swiglu``: w's rows are [gate; up]; the result has N/2 columns of silu(gate) * up, or of the
    clamped gate (csrc/common/gated.cuh) when ``gate_limit`` is positive."""
    _lib.require_cuda_tensor(x, w.w)
    assert x.dtype == torch.bfloat16 and x.dim() == 2 and x.stride(1) == 1
    m, k = x.shape
    n = w.n
    assert k == w.k
    e = w.experts if offsets is not None else 0
    if offsets is not None:
        assert offsets.dtype == torch.int32 and offsets.numel() == e + 1
    if out is None:
        out = torch.empty(m, n // 2 if swiglu else n, dtype=torch.bfloat16, device=x.device)
    # the epilogue reads the residual with the result's row stride
    assert residual is None or (residual.dim() == 2 and residual.shape[0] >= m and residual.shape[1] >= n and
                                residual.stride(1) == 1 and (m == 1 or residual.stride(0) == out.stride(0)))
    route = tiles_route(w, m, e, swiglu) if bn == 0 else "tiles"
    if route == "row" and row_supported(x, w, out, residual, swiglu) and \
            (residual is None or (e == 0 and not swiglu and residual.stride(0) == out.stride(0))):
        return row_gemm(x, w, residual, out, offsets, swiglu, gate_limit, pdl)
    if bn == 0 and (route == "pair" or tiles_route(w, m, e, swiglu, row=False) == "pair") and (residual is None or (e == 0 and not swiglu)) and \
            _pair_ready(x, out, residual) and out.dtype == torch.bfloat16:
        return pair_gemm(x, w, residual, out, offsets, swiglu, gate_limit, pdl)
    rc = _lib.cuda().rmlx_xgemm(w.kind, x.data_ptr(), w.w.data_ptr(), _lib.ptr(w.scales),
                                _lib.ptr(w.biases), out.data_ptr(), _lib.ptr(residual),
                                _lib.ptr(offsets), e, m, n, k, x.stride(0), out.stride(0), bn, int(swiglu),
                                gate_limit,
                                GemmStatus.get(x.device).data_ptr(), int(pdl), _lib.stream_ptr())
    _lib.check(rc, "xgemm")
    return out


def tiles_route(w: LinearWeight, m: int, experts: int = 0, swiglu: bool = False, row: bool = True) -> str:
    """The kernel that ``xgemm`` prefers for m rows whose operands and results lie on 16-byte rows: "row", "pair" or "tiles"."""
    n, k = w.n, w.k
    q4 = w.kind == W_Q4
    if row and q4 and not w.scales_f16 and row_pays(m, n, k, experts) and n % 128 == 0 and k % 512 == 0:
        return "row"
    if m > 128 and pair_pays(w.kind, m, n, k, experts) and (not swiglu or n % 256 == 0) and k % 8 == 0 and \
            (not q4 or (not w.scales_f16 and k % 512 == 0)):
        return "pair"
    return "tiles"


def row_tables_ready(w: LinearWeight) -> bool:
    """Whether the copies of ``rmlx_row_gemm`` can read a 4-bit weight's tables."""
    return ((w.w.data_ptr() | w.scales.data_ptr() | w.biases.data_ptr()) % 16 == 0 and
            w.w.is_contiguous() and w.scales.is_contiguous() and w.biases.is_contiguous())


def row_pays(m: int, n: int, k: int, experts: int = 0) -> bool:
    """Whether 4-bit weights go to the kernel whose 128 product rows are rows of W and whose columns are the rows of x that there are
    (csrc/kernels/row_gemm.cu), rather than to tiles of 128 or 256 rows of x.

    Experts (time of both projections against the tiles', rows of x per expert): 128 of 4096 x 1536 0.6 to 0.7 from 9 to 64 rows, 0.87 at 96,
    0.69 at 128, 0.88 at 176; 32 of 2048 x 2048 0.6, 0.87, 1.01, 0.82, 0.97; 64 of 2048 x 1024 0.6, 0.87, 1.0, 0.85, 1.04. From 192 rows on, where
    a pair of SMs takes the tiles (whole ones of 256 columns), 1.25, 1.39, 1.48. Small experts have too few tiles of W to keep all SMs busy: 16 of
    1024 x 512 0.94 at 32 rows and 1.4 at 160, 16 of 1024 x 1024 1.1 at 96 and 1.16 at 176, 32 of 1024 x 512 1.27 and 1.28; but not those of long K, 8 of
    4096 x 7168 0.69 and 0.82.
    One weight (us, this kernel / the tiles, at 33, 64 and 96 rows). Up to 9472 rows of W the tiles of x's rows are one round of the SMs and their
    time is K's, while this kernel shares K between blocks at a cost that grows with the rows: 8192 x 2048 16 / 15, 19 / 15, 22 / 15; 8192 x 3072 18 /
    20, 21 / 20, 25 / 20; 8192 x 4096 20 / 25, 23 / 25, 27 / 25; 8192 x 5120 22 / 30, 25 / 30, 29 / 30; half as wide it has twice the blocks: 4096 x 2048
    13 / 14, 14 / 14, 16 / 14, 4096 x 3072 15 / 19, 16 / 19, 19 / 20. Then the tiles take two rounds: 9728 x 1024 11 / 15, 11 / 14, 13 / 14; 12288 x
    4096 23 / 45, 24 / 45, 25 / 46. From 14336 on they are twice as wide: 16384 x 1024 12 / 13, 13 / 12, 14 / 12; x 1536 14 / 17, 14 / 15, 16 / 15; x
    2048 16 / 18, 16 / 18, 18 / 18; and from 28672 on both read at the memory's rate, or for small K write at it: 32768 x 1024 16 / 16, 17 / 16, 20 /
    16; x 2048 24 / 23, 25 / 24, 26 / 24; x 3072 32 / 32, 32 / 32, 34 / 33; x 4096 39 / 40, 40 / 41, 42 / 42; 65536 x 4096 69 / 74, 71 / 75, 73 / 77."""
    if experts:
        return (m < 192 * experts or (n % 256 != 0 and m <= 256 * experts)) and (m <= 32 * experts or experts * n * k >= 1 << 26)
    if n * k < 1 << 23:
        return False
    if n <= 4096:
        most = 72 if k < 3072 else 96
    elif n <= 9472:
        most = 3 * k // 128 - 24
    elif n < 14336:
        most = 96
    elif n <= 24576:
        most = 0 if k < 1024 else 32 if k < 1536 else 64 if k < 2048 else 96
    else:
        most = 0 if k < 1024 else 32 if k < 2560 else 64 if k < 4096 else 96
    return m <= min(most, 96)


def row_supported(x: torch.Tensor, w: LinearWeight, out: torch.Tensor, residual: Optional[torch.Tensor] = None,
                  swiglu: bool = False) -> bool:
    """What ``rmlx_row_gemm`` asks of its operands: bf16 scales, 16-byte rows of x, results on 4 bytes."""
    return (not w.scales_f16 and x.data_ptr() % 16 == 0 and out.data_ptr() % 4 == 0 and out.stride(1) == 1 and
            (residual is None or (residual.data_ptr() % 4 == 0 and out.dtype == torch.bfloat16)) and
            row_tables_ready(w) and
            bool(_lib.cuda().rmlx_row_gemm_supported(w.n, w.k, x.stride(0), out.stride(0), int(swiglu))))


def row_gemm(x: torch.Tensor, w: LinearWeight, residual: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
             offsets: Optional[torch.Tensor] = None, swiglu: bool = False, gate_limit: float = 0.0, pdl: bool = False,
             out_dtype=torch.bfloat16, split: int = 0) -> torch.Tensor:
    """``xgemm`` with 4-bit weights on csrc/kernels/row_gemm.cu; fp32 results are the accumulators as they are. ``split``: blocks that
    share K (1, 2, 4, 8; 0: chosen; experts: 1)."""
    _lib.require_cuda_tensor(x, w.w)
    assert x.dtype == torch.bfloat16 and x.dim() == 2 and x.stride(1) == 1 and w.kind == W_Q4
    m, k = x.shape
    n = w.n
    assert k == w.k
    e = w.experts if offsets is not None else 0
    if offsets is not None:
        assert offsets.dtype == torch.int32 and offsets.numel() == e + 1
    if out is None:
        out = torch.empty(m, n // 2 if swiglu else n, dtype=out_dtype, device=x.device)
    assert out.dtype in (torch.bfloat16, torch.float32) and out.shape[0] >= m and out.shape[1] >= (n // 2 if swiglu else n)
    assert residual is None or (residual.dtype == torch.bfloat16 and residual.shape[0] >= m and residual.shape[1] >= n and
                                residual.stride(1) == 1 and (m == 1 or residual.stride(0) == out.stride(0)))
    rc = _lib.cuda().rmlx_row_gemm(x.data_ptr(), w.w.data_ptr(), w.scales.data_ptr(), w.biases.data_ptr(), out.data_ptr(),
                                   int(out.dtype == torch.float32), _lib.ptr(residual), _lib.ptr(offsets), e, m, n, k, x.stride(0),
                                   out.stride(0), int(swiglu), gate_limit, split, GemmStatus.get(x.device).data_ptr(), int(pdl),
                                   _lib.stream_ptr())
    _lib.check(rc, "row_gemm")
    return out


def pair_pays(kind: int, m: int, n: int, k: int, experts: int = 0) -> bool:
    """Whether 256 x 256 tiles of SM pairs are faster than 128-row tiles of single SMs.

    Measured (us, pairs / single SMs). 4-bit, 2048 rows: 28672 x 4096 346 / 455, 9216 x 4096 109 / 150, 4096 x 14336 176 / 243; 512
    rows: 102 / 147, 34 / 44, 82 / 93, 4096 x 4096 (32 tiles) 31 / 31; 256 rows: 4096 x 4096 29 / 28. bf16, 8192 x 28672 x 4096 1232 /
    1371, 1024 x 4096 x 4096 (64 tiles) 29 / 31, 512 x 9216 x 4096 (72) 32 / 39, 512 x 4096 x 8192 (32) 52 / 43. 4-bit experts (128 of
    3072 x 4096 and 4096 x 1536): 930 + 560 / 1026 + 612 at 256 rows each, 622 + 369 / 626 + 376 at 128, where half of a pair's rows
    are mostly empty."""
    if experts:
        return kind == W_Q4 and m >= 192 * experts and n % 256 == 0
    tiles = -(-m // 256) * -(-n // 256)
    return n % 32 == 0 and (m > 128 and tiles >= 32 if kind == W_Q4 else tiles >= 60 and m > 128)


def _pair_ready(x: torch.Tensor, out: torch.Tensor, residual: Optional[torch.Tensor]) -> bool:
    """16-byte rows, as the pair kernel loads and stores them."""
    return x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and out.stride(0) % 8 == 0 and out.data_ptr() % 16 == 0 and \
        out.stride(1) == 1 and (residual is None or (residual.data_ptr() % 16 == 0 and residual.shape == out.shape))


def pair_gemm(x: torch.Tensor, w: LinearWeight, residual: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
              offsets: Optional[torch.Tensor] = None, swiglu: bool = False, gate_limit: float = 0.0, pdl: bool = False) -> torch.Tensor:
    """``xgemm`` on 256 x 256 tiles of SM pairs (csrc/kernels/pair_gemm.cu)."""
    _lib.require_cuda_tensor(x, w.w)
    assert x.dtype == torch.bfloat16 and x.dim() == 2 and x.stride(1) == 1
    m, k = x.shape
    n = w.n
    assert k == w.k
    e = w.experts if offsets is not None else 0
    if offsets is not None:
        assert offsets.dtype == torch.int32 and offsets.numel() == e + 1
    if out is None:
        out = torch.empty(m, n // 2 if swiglu else n, dtype=torch.bfloat16, device=x.device)
    if residual is not None:
        assert residual.shape == out.shape and residual.stride() == out.stride()
    rc = _lib.cuda().rmlx_pair_gemm(w.kind, x.data_ptr(), w.w.data_ptr(), _lib.ptr(w.scales), _lib.ptr(w.biases), out.data_ptr(),
                                    _lib.ptr(residual), _lib.ptr(offsets), e, m, n, k, x.stride(0), out.stride(0), int(swiglu),
                                    gate_limit, GemmStatus.get(x.device).data_ptr(), int(pdl), _lib.stream_ptr())
    _lib.check(rc, "pair_gemm")
    return out


def qmm(x: torch.Tensor, w: LinearWeight, residual: Optional[torch.Tensor] = None,
        out: Optional[torch.Tensor] = None, pdl: bool = False) -> torch.Tensor:
    """x @ W^T for affine-quantised W: a few rows go through the weight-streaming kernel (``ops/narrow.py``); otherwise 4-bit
    weights are expanded inside the tensor-core GEMM's main loop; 8-bit weights, weights with fp16 scales and 4-bit shapes the
    fused kernel does not take are expanded to bf16 by the dequantisation kernel first and go through the bf16 tensor-core GEMM."""
    assert w.kind != 0
    if x.shape[0] <= 64 and narrow.pays(w, x.shape[0]) and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and \
            (residual is None or narrow.same_layout(residual, out, x.shape[0], w.n)):
        return narrow.narrow_gemm(x, w, residual=residual, out=out, pdl=pdl)
    if w.kind == W_Q4 and not w.scales_f16 and _lib.cuda().rmlx_qgemm_supported(w.k):
        return xgemm(x, w, residual, out, pdl=pdl)
    return gemm_bf16(x, w.dense_bf16(), residual=residual, out=out, pdl=pdl)
