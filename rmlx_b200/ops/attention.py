"""Prompt-phase attention over the paged KV cache. Two kernels: the tcgen05 one
(csrc/kernels/flash_prefill_tc.cu; head_dim 128, optional sliding window) and the mma.sync one
(csrc/kernels/flash_prefill.cu; every other shape). The decode-phase kernel is
``ops.decode.flash_decode_paged``. Counterpart of the reference's sdpa prefill kernels
(crates/rmlx-core/src/ops/sdpa.rs:1873-2855), reading pages in place."""
from __future__ import annotations

import math
import os
from typing import Optional

import torch

from .. import _lib
from . import decode
from .gemm import GemmStatus

_lib.register_cuda_sigs({
    "rmlx_flash_prefill_paged": ("pppppiiiiiifip", "i"),
    "rmlx_flash_prefill_tc_supported": ("ii", "i"),
    "rmlx_flash_prefill_tc": ("pppppiiiiiiifipip", "i"),
})


def prefill_kernel_choice(head_dim: int, window: int) -> str:
    """Which kernel ``flash_prefill_paged`` runs for this shape: ``"tc"`` (tcgen05), or ``"mma"``.
    ``RMLX_FLASH_PREFILL=mma`` forces the mma.sync kernel."""
    if (os.environ.get("RMLX_FLASH_PREFILL", "tc") != "mma"
            and _lib.cuda().rmlx_flash_prefill_tc_supported(head_dim, window)):
        return "tc"
    return "mma"


#: query rows up to which a prompt portion attends on the decode kernel, each row a sequence of its own length over the same pages: five rows
#: over 1000 keys of 16/4 heads 8 us, 22 on the prompt kernel, whose blocks walk all keys one after another; and an 8-bit cache is read as it is
FEW_ROWS = 8


def few_rows_plan(t: int, hq: int, hkv: int, head_dim: int, tokens: int, q8: bool) -> int:
    """The cluster plan for ``t`` last rows of a sequence of ``tokens``; 0: the prompt kernels, which also take them where the decode
    kernel is switched off (``RMLX_FLASH_DECODE_CLUSTER=0``) or ``RMLX_FLASH_PREFILL=mma`` names one of theirs."""
    if t > FEW_ROWS or head_dim not in (64, 128) or not decode._FD_CLUSTER or os.environ.get("RMLX_FLASH_PREFILL", "tc") == "mma":
        return 0
    # heads of 64 over few keys: the prompt kernel needs no merge (us, 2.6 / 3.4 at 24 keys, 4.4 / 4.7 at 100, 13.9 / 5.2 at 500)
    if head_dim == 64 and tokens <= 128 and not q8:
        return 0
    tiles = t * hkv * _lib.cuda().rmlx_flash_decode_gtiles(hq, hkv)
    return decode.cluster_plan(t, hq, hkv, head_dim, tokens, q8, tiles) if decode.clusters_pay(tiles, head_dim, tokens, q8) else 0


def few_rows_attention(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, block_row: torch.Tensor, lens: torch.Tensor, plan: int,
                       scale: float, window: int = 0, k_sb: Optional[torch.Tensor] = None, v_sb: Optional[torch.Tensor] = None) -> torch.Tensor:
    """q [T, Hq, D]: row i attends to the first ``lens[i]`` keys of the one sequence whose pages ``block_row`` lists."""
    t, hq, d = q.shape
    out = torch.empty_like(q)
    rc = _lib.cuda().rmlx_flash_decode_cluster(
        q.data_ptr(), k_cache.data_ptr(), _lib.ptr(k_sb), v_cache.data_ptr(), _lib.ptr(v_sb), block_row.data_ptr(), lens.data_ptr(),
        out.data_ptr(), t, hq, k_cache.shape[1], d, block_row.numel(), 0, plan, window, scale, 0, 0, _lib.stream_ptr())
    _lib.check(rc, "flash_decode_cluster")
    return out


def flash_prefill_paged(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                        block_row: torch.Tensor, pos0: int, scale: Optional[float] = None,
                        window: int = 0, out: Optional[torch.Tensor] = None,
                        pdl: bool = False) -> torch.Tensor:
    """q [T, Hq, D] bf16 at positions pos0..pos0+T-1 of one sequence whose pages (already holding
    keys/values 0..pos0+T-1) are listed in ``block_row`` (int32, device). Causal; ``window`` > 0
    limits each query to the last ``window`` keys."""
    _lib.require_cuda_tensor(q, k_cache, v_cache, block_row)
    t, hq, d = q.shape
    assert q.is_contiguous() and q.dtype == torch.bfloat16 and block_row.dtype == torch.int32
    assert k_cache.shape[2] == 16 and k_cache.shape[3] == d
    assert k_cache.is_contiguous() and v_cache.is_contiguous() and k_cache.shape == v_cache.shape
    assert block_row.numel() * 16 >= pos0 + t
    if scale is None:
        scale = 1.0 / math.sqrt(d)
    if out is None:
        out = torch.empty_like(q)
    kind = prefill_kernel_choice(d, window)
    if kind == "mma":
        rc = _lib.cuda().rmlx_flash_prefill_paged(
            q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), block_row.data_ptr(),
            out.data_ptr(), t, hq, k_cache.shape[1], d, pos0, window, scale, int(pdl),
            _lib.stream_ptr())
    else:
        rc = _lib.cuda().rmlx_flash_prefill_tc(
            q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), block_row.data_ptr(),
            out.data_ptr(), t, hq, k_cache.shape[1], d, k_cache.shape[0], pos0, int(window or 0), scale,
            int(os.environ.get("RMLX_FLASH_PREFILL_LANES", "0")),     # query tiles per CTA: 1, 2, 0 = choose
            GemmStatus.get(q.device).data_ptr(), int(pdl), _lib.stream_ptr())
    _lib.check(rc, "flash_prefill_paged")
    return out
