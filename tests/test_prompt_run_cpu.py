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
