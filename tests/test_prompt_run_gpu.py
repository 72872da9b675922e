"""A prompt portion from one native call (csrc/runtime/prompt_run.cu) against the same launches made one by one: the same kernels on the
same values, so logits and cache are the same to the bit."""
import pytest
import torch

from rmlx_b200.config import FeedForwardType, MoeConfig, TransformerConfig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda")


def _model(dev, experts, quant, window=0, hd=128, bias=False, expert=(1024, 512), top=2):
    from rmlx_b200.models.transformer import TransformerModel
    from rmlx_b200.models.weights import LayerWeights, ModelWeights, ParallelLayout
    from rmlx_b200.ops.weights import LinearWeight
    g = torch.Generator(device=dev).manual_seed(1)
    d, inner, vocab = (*expert, 2048) if experts else (2048, 4096, 2048)
    hq, hkv = d // hd, d // hd // 4
    ff = FeedForwardType.moe_(MoeConfig(experts, top, d, inner)) if experts else FeedForwardType.gated(inner)
    cfg = TransformerConfig(hidden_size=d, num_heads=hq, num_kv_heads=hkv, head_dim=hd, num_layers=2, vocab_size=vocab, max_seq_len=2048,
                            rope_theta=1e4, ff_type=ff, sliding_window=window, name="prompt-run").validate()

    def lin(n, k, e=0):
        return LinearWeight.random(n, k, quant, dev, experts=e, generator=g)

    def norm():
        return (1 + 0.1 * torch.randn(d, device=dev, generator=g)).to(torch.bfloat16)

    layers = []
    for _ in range(2):
        ff_w = {"w_gate_up": lin(2 * inner, d), "w_down": lin(d, inner)} if not experts else {
            "router": torch.randn(experts, d, device=dev, generator=g).mul_(0.1).to(torch.bfloat16),
            "experts_gate_up": lin(2 * inner, d, experts), "experts_down": lin(d, inner, experts),
            "expert_bias": torch.randn(experts, device=dev, generator=g) * 0.1 if bias else None}
        layers.append(LayerWeights(norm1=norm(), wqkv=lin((hq + 2 * hkv) * hd, d), wo=lin(d, hq * hd), norm2=norm(), **ff_w))
    embed = torch.randn(vocab, d, device=dev, generator=g).to(torch.bfloat16)
    return TransformerModel(ModelWeights(cfg=cfg, layout=ParallelLayout(), embed=embed, layers=layers, final_norm=norm(), lm_head=lin(vocab, d)))


def _prompts(model, lens, kv, at_once):
    """Portions of one sequence after one another: logits of each, and the cache."""
    from rmlx_b200.models.prefill import enable_native_prefill
    assert enable_native_prefill(model)
    run = model._native_prefill.at_once.run
    calls = []

    def traced(*args):
        h = run(*args) if at_once else None
        calls.append(h is not None)
        return h

    model._native_prefill.at_once.run = traced
    cache = model.new_cache(sum(lens) // 16 + 3, max_seqs=1, kv_quant=kv)
    cache.add_sequence(0)
    g = torch.Generator().manual_seed(2)
    out = []
    for n in lens:
        ids = torch.randint(0, model.cfg.vocab_size, (n,), generator=g).to(model.device)
        out.append(model.prefill(ids, cache, 0, all_logits=n <= 40))
    assert all(c == at_once for c in calls) and cache.seq_len(0) == sum(lens)
    pools = [*cache.k, *cache.v] + ([*cache.k_sb, *cache.v_sb] if kv else [])
    return out, [p.clone() for p in pools]


@pytest.mark.parametrize("experts", [0, 16])
@pytest.mark.parametrize("quant", ["q4", "q8", None])
@pytest.mark.parametrize("kv,window,hd", [(None, 0, 128), ("q8", 300, 128), (None, 0, 64)])
def test_same_as_launch_by_launch(dev, experts, quant, kv, window, hd):
    # portions on each side of the lines between the projections' kernels
    lens = [1, 5, 8, 9, 17, 33, 40, 90, 100, 300, 700, 6]
    res = [_prompts(_model(dev, experts, quant, window, hd, bias=hd == 64), lens, kv, at_once) for at_once in (False, True)]
    for a, b in zip(res[0][0] + res[0][1], res[1][0] + res[1][1]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("quant,top,lens", [("q8", 1, [193, 256, 448]), ("q8", 2, [192, 193, 224]), ("q4", 1, [193, 384])])
def test_few_rows_per_expert_of_a_longer_portion(dev, quant, top, lens):
    """More rows than the router takes along and few for each expert: norm, logits and selection as launches of their own, then the experts
    on the weight-streaming kernel."""
    from rmlx_b200.models.prefill import ROUTER_ROWS
    from rmlx_b200.ops import narrow
    res = []
    for at_once in (False, True):
        model = _model(dev, 32, quant, expert=(2048, 1024), top=top)
        up, down = model.w.layers[0].experts_gate_up, model.w.layers[0].experts_down
        assert max(lens) > ROUTER_ROWS and all(narrow.pays_grouped(up, down, t * top) for t in lens)
        res.append(_prompts(model, lens, None, at_once))
    for a, b in zip(res[0][0] + res[0][1], res[1][0] + res[1][1]):
        assert torch.equal(a, b)


def test_router_at_an_odd_address(dev):
    """A router that no kernel reads raises from the native call as it does launch by launch."""
    from rmlx_b200 import _lib
    for at_once in (False, True):
        model = _model(dev, 16, "q4")
        r = model.w.layers[1].router
        odd = torch.empty(r.numel() + 1, dtype=r.dtype, device=dev)[1:].view_as(r)
        odd.copy_(r)
        model.w.layers[1].router = odd
        for n in (5, 300):
            with pytest.raises(_lib.NativeError):
                _prompts(model, [n], None, at_once)


def test_not_covered(dev):
    """Weights that change between two portions are taken as they are; rows of W apart go launch by launch."""
    from rmlx_b200.ops.weights import LinearWeight, W_BF16
    model = _model(dev, 0, None)
    first = _prompts(model, [40], None, True)[0][0]
    wide = torch.zeros(model.w.layers[0].wqkv.n, model.cfg.hidden_size + 64, dtype=torch.bfloat16, device=dev)
    wide[:, :model.cfg.hidden_size] = model.w.layers[0].wqkv.w
    model.w.layers[0].wqkv = LinearWeight(W_BF16, wide[:, :model.cfg.hidden_size])
    assert model._native_prefill.at_once._plain(model.w.layers[0].wqkv, 40) == 0
    assert float((_prompts(model, [40], None, False)[0][0] - first).norm() / first.norm()) < 1e-2
    model.w.layers[0].wqkv = LinearWeight(W_BF16, wide[:, :model.cfg.hidden_size].contiguous() * 2)
    assert not torch.equal(_prompts(model, [40], None, True)[0][0], first)


def test_host_ids_raise(dev):
    """Ids on the host (the attached path called directly) raise before anything is launched, and the model goes on working."""
    from rmlx_b200 import _lib
    from rmlx_b200.models.prefill import NativePrefill
    model = _model(dev, 0, "q4")
    native, cache = NativePrefill(model), model.new_cache(8, max_seqs=1)
    cache.add_sequence(0)
    ids = torch.arange(20, dtype=torch.int32)
    assert native.at_once.run(ids, cache, 0, 0) is None
    with pytest.raises(_lib.NativeError):
        native(ids, cache, 0)
    assert torch.isfinite(native(ids.to(dev), cache, 0)).all()


@pytest.mark.parametrize("experts", [0, 16])
@pytest.mark.parametrize("quant", ["q4", "q8", None])
@pytest.mark.parametrize("kv", [None, "q8"])
def test_block_is_what_the_plan_counts(dev, experts, quant, kv):
    """The block that a portion allocates is never more than the static plan says, and a long portion's is the plan's to the byte."""
    from rmlx_b200.models.prefill import NativePrefill
    from rmlx_b200.models.prefill_plan import PrefillPlan
    model = _model(dev, experts, quant)
    native, cache = NativePrefill(model), model.new_cache(80, max_seqs=1, kv_quant=kv)
    cache.add_sequence(0)
    for t in (1, 7, 40, 100, 700):
        at = cache.seq_len(0)
        cache.reserve(0, t)
        h = native.at_once.run(torch.zeros(t, dtype=torch.int32, device=dev), cache, 0, at)
        cache.commit(0, t)
        plan = PrefillPlan(model.cfg, t, weights=quant or "bf16", kv_quant=kv, context=at + t).scratch_bytes
        assert h.untyped_storage().nbytes() <= plan
    assert h.untyped_storage().nbytes() == plan


def test_tables_of_numbers_come_with_the_path(dev):
    """They are there for every position of the model when the path is attached; no portion within its length makes new ones."""
    from rmlx_b200.models.prefill import NativePrefill
    model = _model(dev, 0, "q4")
    native, cache = NativePrefill(model), model.new_cache(130, max_seqs=1)
    cache.add_sequence(0)
    made = list(native.at_once._numbers)
    assert len(made) == 1 and made[0][0].numel() == model.cfg.max_seq_len + 1
    for t in (1, model.cfg.max_seq_len - 1):
        native(torch.zeros(t, dtype=torch.int32, device=dev), cache, 0)
    assert len(native.at_once._numbers) == 1 and native.at_once._numbers[0] is made[0]
    assert torch.equal(made[0][0], torch.arange(model.cfg.max_seq_len + 1, dtype=torch.int32, device=dev)) and not made[0][1].any()
