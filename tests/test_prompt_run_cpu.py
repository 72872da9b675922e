"""What a prompt portion's native call (models/prefill.py) refuses and plans before anything is launched, on the CPU."""
import pytest
import torch

from rmlx_b200 import _lib
from rmlx_b200.config import FeedForwardType, TransformerConfig


class _Kernels:
    """Stands in for the kernel library: notes what was launched and finds nothing wrong."""

    def __init__(self, real):
        self.called = []
        self.rmlx_prompt_sizes = real.rmlx_prompt_sizes

    def __getattr__(self, name):
        def call(*args):
            self.called.append(name)
            return 0
        return call


def _model():
    from rmlx_b200.models.transformer import TransformerModel
    from rmlx_b200.models.weights import from_state_dict, random_state_dict
    cfg = TransformerConfig(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=64, num_layers=2, vocab_size=128, max_seq_len=128,
                            ff_type=FeedForwardType.gated(512)).validate()
    return TransformerModel(from_state_dict(cfg, random_state_dict(cfg, 0)))


@pytest.mark.parametrize("ids", [torch.arange(9), torch.arange(9, dtype=torch.int32)])
def test_host_tensors_raise_before_any_launch(monkeypatch, ids):
    """Host memory must not reach a kernel by its address: token ids (and with them the model and the cache) on the host raise what the
    launches one by one raise."""
    from rmlx_b200.models.prefill import NativePrefill, PromptRun
    from rmlx_b200.ops.gemm import GemmStatus
    model, lib = _model(), _Kernels(_lib.cuda())
    cache = model.new_cache(4, max_seqs=1)
    cache.add_sequence(0)
    word = torch.zeros(64, dtype=torch.int32)
    monkeypatch.setattr(_lib, "cuda", lambda: lib)
    monkeypatch.setattr(_lib, "stream_ptr", lambda *a: 0)
    monkeypatch.setattr(GemmStatus, "get", classmethod(lambda cls, device: word))
    monkeypatch.setattr(PromptRun, "_tables", lambda self, n: (word, word))
    native = NativePrefill(model)
    with pytest.raises(_lib.NativeError):
        native(ids, cache, 0)
    assert not [name for name in lib.called if name in ("rmlx_prompt_run", "rmlx_embedding")]


def test_few_rows_follow_the_kernel_switches(monkeypatch):
    """Portions of up to eight rows attend on the decode kernel, unless the switch of that kernel is off or the one of the prompt kernels
    names its ``mma.sync`` form."""
    from rmlx_b200.ops import attention, decode

    class _Plans:
        rmlx_flash_decode_gtiles = staticmethod(lambda hq, hkv: 1)
        rmlx_flash_decode_cluster_plan = staticmethod(lambda batch, tiles, tokens, hd, q8: 4 << 16 | tiles)

    monkeypatch.setattr(_lib, "cuda", _Plans)
    monkeypatch.delenv("RMLX_FLASH_PREFILL", raising=False)
    monkeypatch.setattr(decode, "_FD_CLUSTER", True)

    def plan(t=5):
        return attention.few_rows_plan(t, 16, 4, 128, 1000, False)

    assert plan() == 4 << 16 | 20 and plan(8) and plan(9) == 0 and attention.few_rows_plan(5, 16, 4, 96, 1000, False) == 0
    monkeypatch.setenv("RMLX_FLASH_PREFILL", "mma")
    assert plan() == 0
    monkeypatch.setenv("RMLX_FLASH_PREFILL", "tc")
    assert plan()
    monkeypatch.setattr(decode, "_FD_CLUSTER", False)
    assert plan() == 0


# ---------------------------------------------------------------------------------------------- work space
def _launches(moe, inside, mid, kv, expanded):
    """(reads, writes) of a layer's launches in their order; ``inside``: the norms run within the next product."""
    def linear(x, out, *more):
        return ([([], ["dense"]), (["dense", x, *more], [out])] if expanded else [([x, *more], [out])])

    def normed(h, out):
        return [([h], [out])] if inside else [([h], ["xn"]), *linear("xn", out)]

    seq = [*normed("h0", "qkv"), (["qkv"], ["q"])]
    seq += [([], ["kk"]), ([], ["vv"]), (["q", "kk", "vv"], ["attn"])] if kv else [(["q"], ["attn"])]
    seq += linear("attn", "h1", "h0")
    if not moe:
        seq += normed("h1", "mid") + [(["mid"], ["act"])] if mid else normed("h1", "act")
        return seq + linear("act", "h0", "h1")
    if inside:
        seq += [(["h1"], ["logits"]), (["logits"], ["idx", "wts"])]
    else:
        seq += [(["h1"], ["xn"]), (["xn"], ["logits"]), (["logits"], ["idx", "wts", "counts", "offsets"])]
    if moe == "tiles":
        return seq + [(["xn", "idx", "offsets"], ["cursors", "xs", "row_of"]), (["xs", "offsets"], ["act"]), (["act", "offsets"], ["y"]),
                      (["y", "row_of", "wts", "h1"], ["h0"])]
    rows = "h1" if inside else "xn"
    return seq + [(["idx"], ["offsets", "order"]), ([rows, "order", "offsets"], ["act"]), (["act", "order", "offsets"], ["y"]),
                  (["y", "idx", "wts", "h1"], ["h0"])]


@pytest.mark.parametrize("moe,inside,mid,kv,expanded", [
    (None, False, False, False, False), (None, True, False, False, False), (None, False, True, True, True), (None, False, True, False, False),
    ("tiles", False, False, True, True), ("tiles", False, False, False, False), ("narrow", True, False, False, False),
    ("narrow", False, False, True, False)])
def test_work_space_holds_what_is_still_read(moe, inside, mid, kv, expanded):
    """Through two layers, no launch writes where a piece lies that it or a later launch still reads; and the block is shorter than its
    pieces side by side."""
    from rmlx_b200.models.prefill_plan import PIECES, prompt_block
    seq = [([], ["h0"])] + 2 * _launches(moe, inside, mid, kv, expanded) + [(["h0"], [])]
    used = {name for reads, writes in seq for name in (*reads, *writes)}
    sizes = {name: 1000 * (i % 7 + 1) + i for i, name in enumerate(PIECES) if name in used}
    at, total = prompt_block(sizes)
    assert set(at) == set(PIECES) and all(a % 256 == 0 and a + sizes.get(n, 0) <= total for n, a in at.items())
    assert total < sum(sizes.values())
    for i, (reads, writes) in enumerate(seq):
        for w in writes:
            for other in used - {w}:
                later = [(other in r, other in o) for r, o in seq[i + 1:]]
                needed = other in reads or other in writes or next((r for r, o in later if r or o), False)
                if needed:
                    assert at[w] + sizes[w] <= at[other] or at[other] + sizes[other] <= at[w], (i, w, other)


def test_plan_counts_the_block():
    """Bytes that a portion takes, in models of the benchmarks' sizes; the chunk keeps them within the limit it is given."""
    from rmlx_b200.config import MoeConfig, moe_a22b_config
    from rmlx_b200.models.prefill import plan_chunk
    from rmlx_b200.models.prefill_plan import PrefillPlan, prompt_block
    from rmlx_b200.models.weights import ParallelLayout
    mb = 2 ** 20
    dense = TransformerConfig(hidden_size=4096, num_heads=32, num_kv_heads=8, head_dim=128, num_layers=1, vocab_size=128,
                              ff_type=FeedForwardType.gated(14336)).validate()
    # residual stream twice, normed rows, gated rows
    assert PrefillPlan(dense, 8192).scratch_bytes == (2 * 64 + 64 + 224) * mb
    # 8-bit weights: both halves of the gate before the product, and the widest weight in bf16
    assert PrefillPlan(dense, 8192, weights="q8").scratch_bytes == (2 * 64 + 64 + 224 + 448 + 28672 * 4096 * 2 // mb) * mb
    # 8-bit cache, a short portion of a long context: queries, qkv, and both sides of the pages
    assert PrefillPlan(dense, 512, kv_quant="q8", context=65536).scratch_bytes == (2 * 4 + 4 + 6 + 2 * 128) * mb
    moe = PrefillPlan(moe_a22b_config(2), 8192)
    d, top, inner = (moe.cfg.hidden_size, moe.cfg.ff_type.moe.num_experts_per_token, moe.cfg.ff_type.moe.intermediate_dim)
    assert 0 <= moe.scratch_bytes - 8192 * (3 * d + top * (inner + d)) * 2 < 2 * mb
    assert PrefillPlan(moe_a22b_config(2), 8192, ParallelLayout(0, 2)).scratch_bytes == sum(PrefillPlan(
        moe_a22b_config(2), 8192, ParallelLayout(0, 2)).pieces.values())

    class _M:
        cfg, layout = moe_a22b_config(2), ParallelLayout()

    for limit in (256 * mb, 700 * mb, 4096 * mb):
        chunk = plan_chunk(_M, limit)
        assert prompt_block(PrefillPlan(_M.cfg, chunk, _M.layout).pieces)[1] <= limit
        assert chunk == 8192 or PrefillPlan(_M.cfg, chunk + 128, _M.layout).scratch_bytes > limit
