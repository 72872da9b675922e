"""What this framework is timed on: decode steps and prompts of its transformer, through the entry points a program calls.

A case is one decode step of a batch of sequences (``make_decode_engine`` / ``step``) or one prompt portion (``prefill``) on a
model of a few layers; layers are alike, so a few of them stand for the whole stack. The models are the mixture-of-experts
decoder of ``moe_a22b_config``, the dense and mixture-of-experts decoders of the benchmarks and the tiny dense one of
``tiny_dense_config``. Weights are random, in each of the formats the loaders produce; the residual stream starts
well above what one layer adds, as it is inside a deep stack, and the cache holds N(0, 1) keys and values.
"""
from __future__ import annotations

import math

import torch

from rmlx_b200.config import FeedForwardType, MoeConfig, TransformerConfig
from rmlx_b200.models.transformer import TransformerModel
from rmlx_b200.models.weights import LayerWeights, ModelWeights, ParallelLayout
from rmlx_b200.ops.weights import LinearWeight, W_BF16, W_Q4, W_Q8

DEVICE, PAGE, GROUP, EPS, STD, LONGEST = "cuda", 16, 64, 1e-6, 0.02, 8192

#: width, query heads, key/value heads, head width, inner width, experts, experts per token, vocabulary, rotation base
MODELS = {
    "tiny": (256, 4, 2, 64, 688, 0, 0, 1024, 1e4),
    "dense-2048": (2048, 16, 4, 128, 8192, 0, 0, 32768, 1e4),
    "dense-4096": (4096, 32, 8, 128, 14336, 0, 0, 32768, 1e4),
    "moe-2048": (2048, 16, 4, 128, 2048, 32, 4, 32768, 1e4),
    "moe-4096": (4096, 64, 4, 128, 1536, 128, 8, 151936, 1e6),
}


def _decode(name, model, weights, layers, batch, ctx, kv="bf16", window=0):
    return {"name": name, "path": "decode", "model": model, "weights": weights, "layers": layers, "batch": batch,
            "ctx": ctx, "kv": kv, "window": window}


def _prompt(name, model, weights, layers, tokens, ctx, kv="bf16", window=0, all_logits=False):
    return {"name": name, "path": "prompt", "model": model, "weights": weights, "layers": layers, "tokens": tokens,
            "ctx": ctx, "kv": kv, "window": window, "all_logits": all_logits}


def listed():
    return [
        # the smallest call there is: a two-layer model whose step is launches and latency
        _decode("decode-tiny", "tiny", "bf16", 2, 1, 24),
        # one user talking to the large model: the headline workload
        _decode("decode-moe-q4-x1", "moe-4096", "q4", 4, 1, 4096),
        # a handful of users on one GPU, sequences of different lengths
        _decode("decode-moe-q4-x8", "moe-4096", "q4", 4, 8, 3900),
        # a full serving batch
        _decode("decode-moe-q4-x64", "moe-4096", "q4", 4, 64, 2048),
        # the smaller mixture of experts in 16-bit weights, an odd batch
        _decode("decode-moe-bf16-x5", "moe-2048", "bf16", 4, 5, 777),
        # a dense model in 8-bit weights, a few rows
        _decode("decode-dense-q8-x3", "dense-2048", "q8", 4, 3, 3000),
        # a dense model with 4-bit weights and the 8-bit cache, a middle batch
        _decode("decode-dense-q4-kv8-x16", "dense-4096", "q4", 4, 16, 2000, kv="q8"),
        # a short question to the large model: time to first token
        _prompt("prompt-moe-q4-37", "moe-4096", "q4", 2, 37, 0),
        # an ordinary prompt to the large model
        _prompt("prompt-moe-q4-2048", "moe-4096", "q4", 2, 2048, 0),
        # the longest prompt portion, 16-bit weights
        _prompt("prompt-dense-bf16-8192", "dense-4096", "bf16", 2, 8192, 0),
        # a scheduler's chunk on top of a cached context, 8-bit cache, sliding window
        _prompt("prompt-dense-q4-chunk", "dense-4096", "q4", 2, 512, 3500, kv="q8", window=4096),
        # speculative verification: a few proposed tokens, logits of all of them
        _prompt("prompt-dense-q8-verify", "dense-2048", "q8", 4, 5, 1000, all_logits=True),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    model = rng.choice(["moe-4096", "moe-4096", "moe-2048", "dense-4096", "dense-2048", "tiny"])
    weights = "bf16" if model == "tiny" else rng.choice(["q4", "q4", "q4", "bf16", "q8"])
    if model == "dense-4096" and weights == "q8":
        model = "dense-2048"                             # 8-bit decode steps take inner widths up to about 10000
    longest = 256 if model == "tiny" else LONGEST
    kv = "q8" if model != "tiny" and rng.random() < 0.25 else "bf16"
    window = rng.choice([1024, 4096]) if model.startswith("dense") and rng.random() < 0.25 else 0
    if rng.random() < 0.6:
        batch = _spread(rng, 1, 64)
        if weights == "q8" and 4 <= batch <= 8:
            batch = 3                                    # nor so many rows of the wider projections
        c = _decode("", model, weights, 2, batch, _spread(rng, 16, longest - 64), kv, window)
    else:
        tokens = _spread(rng, 1, 128 if model == "tiny" else 4096)
        ctx = 0 if rng.random() < 0.5 else _spread(rng, 16, longest - tokens)
        c = _prompt("", model, weights, 2, tokens, ctx, kv, window, all_logits=tokens <= 16 and rng.random() < 0.5)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------- inputs
def _lens(case):
    """Tokens in the cache of every sequence: a batch's sequences have different lengths."""
    ctx = case["ctx"]
    return [ctx - (i * 61) % max(1, ctx // 4) for i in range(case.get("batch", 1))]


def _new_tokens(case):
    return case["tokens"] if case["path"] == "prompt" else 1


def _tables(case):
    """Pages of every sequence, in the order in which the cache hands them out: all full pages first, then room for the new
    tokens (page 0 is the cache's own). Returns the tables and the first page that new tokens go to."""
    lens, t = _lens(case), _new_tokens(case)
    tables, at = [], 1
    for n in lens:
        tables.append(list(range(at, at + n // PAGE)))
        at += n // PAGE
    first = at
    for n, row in zip(lens, tables):
        more = -(-(n + t) // PAGE) - n // PAGE
        row += range(at, at + more)
        at += more
    return tables, first, at


class _Maker:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.empty(*shape, dtype=torch.bfloat16, device=DEVICE).normal_(mean, std, generator=self.g)

    def ints(self, high, *shape):
        return torch.randint(0, high, shape, dtype=torch.int64, device=DEVICE, generator=self.g)

    def weight(self, kind, *shape):
        """(codes or values, scales, biases) of a [.., N, K] projection of entries of about STD."""
        if kind == "bf16":
            return self.normal(*shape, std=STD), None, None
        bits = 4 if kind == "q4" else 8
        words = torch.empty(*shape[:-1], shape[-1] * bits // 32, dtype=torch.int32, device=DEVICE)
        words.random_(-(2 ** 31), 2 ** 31 - 1, generator=self.g)
        levels = (1 << bits) - 1
        scales = torch.empty(*shape[:-1], shape[-1] // GROUP, dtype=torch.float32, device=DEVICE)
        # uniform codes: a standard deviation of STD over a range of sqrt(12) of it
        scales.uniform_(0.75, 1.25, generator=self.g).mul_(math.sqrt(12.0) * STD / levels)
        scales = scales.to(torch.bfloat16)
        return words, scales, (-0.5 * levels * scales.float()).to(torch.bfloat16)


def _inputs(case, seed):
    """Everything random of a case, as plain tensors."""
    d, hq, hkv, hd, inner, experts, top, vocab, _ = MODELS[case["model"]]
    mk, kind = _Maker(seed), case["weights"]
    tables, first, pages = _tables(case)
    layers, pools = [], []
    for _ in range(case["layers"]):
        lw = {"norm1": mk.normal(d, std=STD, mean=1.0), "qkv": mk.weight(kind, (hq + 2 * hkv) * hd, d),
              "out": mk.weight(kind, d, hq * hd), "norm2": mk.normal(d, std=STD, mean=1.0)}
        if experts:
            # decided choices: the last chosen expert carries little weight, so a near tie that rounding turns moves the
            # result by no more than rounding does
            lw["router"] = mk.normal(experts, d, std=6.4 * d ** -0.5)
            lw["up"], lw["down"] = mk.weight(kind, experts, 2 * inner, d), mk.weight(kind, experts, d, inner)
        else:
            lw["up"], lw["down"] = mk.weight(kind, 2 * inner, d), mk.weight(kind, d, inner)
        layers.append(lw)
        pool = []
        for _ in range(2):
            if case["kv"] == "q8":
                codes = torch.randint(0, 256, (pages, hkv, PAGE, hd), dtype=torch.uint8, device=DEVICE, generator=mk.g)
                scale = torch.empty(pages, hkv, PAGE, hd // GROUP, device=DEVICE).uniform_(0.75, 1.25, generator=mk.g)
                scale = (scale * math.sqrt(12.0) / 255).to(torch.bfloat16)
                pool.append((codes, torch.stack([scale, (-127.5 * scale.float()).to(torch.bfloat16)], -1)))
            else:
                pool.append((mk.normal(pages, hkv, PAGE, hd), None))
        pools.append(pool)
    return {"layers": layers, "pools": pools, "embed": mk.normal(vocab, d, std=4.0), "norm": mk.normal(d, std=STD, mean=1.0),
            "head": mk.weight(kind, vocab, d), "tokens": mk.ints(vocab, max(len(tables), _new_tokens(case))),
            "tables": tables, "first": first, "pages": pages}


def _config(case):
    d, hq, hkv, hd, inner, experts, top, vocab, theta = MODELS[case["model"]]
    ff = FeedForwardType.moe_(MoeConfig(experts, top, d, inner)) if experts else FeedForwardType.gated(inner)
    return TransformerConfig(hidden_size=d, num_heads=hq, num_kv_heads=hkv, head_dim=hd, num_layers=case["layers"],
                             vocab_size=vocab, max_seq_len=256 if case["model"] == "tiny" else LONGEST, rope_theta=theta,
                             rms_norm_eps=EPS, ff_type=ff, sliding_window=case["window"], name=case["model"]).validate()


# ---------------------------------------------------------------------------------------------- the path
def prepare(case, seed):
    """The loaded model, a cache that holds the sequences so far, the captured decode engine: what a serving process keeps."""
    inp, cfg = _inputs(case, seed), _config(case)
    kind = {"bf16": W_BF16, "q4": W_Q4, "q8": W_Q8}[case["weights"]]

    def lin(t):
        return LinearWeight(kind, *t)

    layers = []
    for lw in inp["layers"]:
        ff = {"router": lw["router"], "experts_gate_up": lin(lw["up"]), "experts_down": lin(lw["down"])} if "router" in lw \
            else {"w_gate_up": lin(lw["up"]), "w_down": lin(lw["down"])}
        layers.append(LayerWeights(norm1=lw["norm1"], wqkv=lin(lw["qkv"]), wo=lin(lw["out"]), norm2=lw["norm2"], **ff))
    model = TransformerModel(ModelWeights(cfg=cfg, layout=ParallelLayout(), embed=inp["embed"], layers=layers,
                                          final_norm=inp["norm"], lm_head=lin(inp["head"])))
    lens, t, tables = _lens(case), _new_tokens(case), inp["tables"]
    cache = model.new_cache(inp["pages"], max_seqs=len(lens), kv_quant="q8" if case["kv"] == "q8" else None)
    for s, n in enumerate(lens):
        cache.add_sequence(s)
        cache.reserve(s, n // PAGE * PAGE)
        cache.commit(s, n // PAGE * PAGE)
    for s, n in enumerate(lens):
        cache.reserve(s, n % PAGE + t)
        cache.commit(s, n % PAGE)
        assert list(cache.manager.block_table(s)) == tables[s]
    for l, pool in enumerate(inp["pools"]):
        for mine, sb, (values, scales) in ((cache.k, cache.k_sb, pool[0]), (cache.v, cache.v_sb, pool[1])):
            mine[l].copy_(values)
            if sb is not None:
                sb[l].copy_(scales)
    # the pages that new tokens go to, as the cache holds them (8-bit cache: their scales)
    held = [p[inp["first"]:] for l in range(case["layers"])
            for p in ((cache.k[l], cache.v[l]) if case["kv"] == "bf16" else (cache.k_sb[l], cache.v_sb[l]))]
    state = {"case": case, "model": model, "cache": cache, "held": held, "lens": lens}
    if case["path"] == "prompt":
        state["tokens"] = inp["tokens"][:t].to(torch.int32)
        model.prefill(state["tokens"][:1], cache, 0)     # attaches the prompt path
        cache.trim(0, 1)
        for l, pool in enumerate(inp["pools"]):
            cache.k[l].copy_(pool[0][0])
            cache.v[l].copy_(pool[1][0])
            if case["kv"] == "q8":
                cache.k_sb[l].copy_(pool[0][1])
                cache.v_sb[l].copy_(pool[1][1])
        return state
    engine = model.make_decode_engine(cache, len(lens))
    engine.bind(range(len(lens)), inp["tokens"].tolist())
    state.update(engine=engine, start=[x.clone() for x in (engine.tokens, engine.positions, engine.seq_lens)])
    engine.step()                                        # records the step, as a serving process does before it serves
    return state


@torch.no_grad()
def run(state):
    """One decode step of the batch, or one prompt portion; both are rolled back first, so that every pass does the same."""
    case, cache = state["case"], state["cache"]
    if case["path"] == "prompt":
        more = cache.seq_len(0) - state["lens"][0]
        if more > 0:
            cache.trim(0, more)
        logits = state["model"].prefill(state["tokens"], cache, 0, all_logits=case["all_logits"])
        return {"logits": logits, "held": state["held"]}
    engine = state["engine"]
    for now, then in zip((engine.tokens, engine.positions, engine.seq_lens), state["start"]):
        now.copy_(then)
    for s, n in enumerate(state["lens"]):
        cache.manager.trim(s, cache.seq_len(s) - n)      # the device's table keeps the row
    engine.step()
    return {"logits": engine.logits[:case["batch"]], "held": state["held"]}


# ---------------------------------------------------------------------------------------------- what it takes
def _attended(case):
    """Pairs of a query and a key that it sees, over all sequences (per head)."""
    t, w = _new_tokens(case), case["window"] or 1 << 40
    return sum(min(w, n + i + 1) for n in _lens(case) for i in range(t))


def _keys_read(case):
    t, w = _new_tokens(case), case["window"] or 1 << 40
    return sum(min(n + t, w + t - 1) for n in _lens(case))


def work(case):
    d, hq, hkv, hd, inner, experts, top, vocab, _ = MODELS[case["model"]]
    rows = _new_tokens(case) * len(_lens(case))
    logits = rows if case["path"] == "decode" or case["all_logits"] else 1
    per = {"bf16": 2.0, "q8": 1.0 + 4.0 / GROUP, "q4": 0.5 + 4.0 / GROUP}[case["weights"]]
    token = 2 * hkv * (hd * 2 if case["kv"] == "bf16" else hd + hd // GROUP * 4)
    attention = d * (hq + 2 * hkv) * hd + hq * hd * d
    used = experts * (1 - (1 - top / experts) ** rows) if experts else 1    # experts that some row chooses
    layer = (attention + used * 3 * inner * d) * per + experts * d * 2 + (_keys_read(case) + rows) * token
    flops = 2 * rows * (attention + (top if experts else 1) * 3 * inner * d + experts * d) + 4 * _attended(case) * hq * hd
    return {"bytes": case["layers"] * layer + vocab * d * per + rows * d * 2 + logits * vocab * 4,
            "flops": case["layers"] * flops + 2.0 * logits * vocab * d}


def tolerance(case):
    # bf16 activations between kernels: up to 0.01 from the 64-bit result
    return {"rel": 0.02, "max": 0.5}


# ---------------------------------------------------------------------------------------------- 64-bit
def _dense(t, kind):
    words, scales, biases = t
    if kind == "bf16":
        return words.double()
    bits = 4 if kind == "q4" else 8
    shifts = torch.arange(0, 32, bits, device=words.device, dtype=torch.int32)
    q = ((words[..., None] >> shifts) & ((1 << bits) - 1)).flatten(-2).double()
    q = q.unflatten(-1, (-1, GROUP))
    return (q * scales.double()[..., None] + biases.double()[..., None]).flatten(-2)


def _norm(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w.double()


def _rotate(x, pos, theta):
    half = x.shape[-1] // 2
    angle = pos.double()[:, None] * theta ** (-torch.arange(half, device=x.device).double() / half)[None]
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _rows(pool, pages, n):
    """The first n cached rows of a sequence, [n, heads, width] in 64 bits."""
    values, sb = pool
    x = values[pages].double()
    if sb is not None:
        sb = sb[pages].double()
        x = (x.unflatten(-1, (-1, GROUP)) * sb[..., :1] + sb[..., 1:]).flatten(-2)
    return x.transpose(1, 2).flatten(0, 1)[:n]


def _attend(q, k, v, start, window):
    """q [T, Hq, D] at positions start.. against k, v [start + T, Hkv, D]."""
    t, hq, hd = q.shape
    share = hq // k.shape[1]
    at, keys = torch.arange(t, device=q.device)[:, None] + start, torch.arange(k.shape[0], device=q.device)[None]
    hidden = keys > at
    if window:
        hidden |= keys <= at - window
    out = torch.empty_like(q)
    for h in range(hq):
        s = (q[:, h] @ k[:, h // share].t()) * hd ** -0.5
        out[:, h] = torch.softmax(s.masked_fill_(hidden, float("-inf")), -1) @ v[:, h // share]
    return out


@torch.no_grad()
def exact(case, seed):
    d, hq, hkv, hd, inner, experts, top, vocab, theta = MODELS[case["model"]]
    inp, kind = _inputs(case, seed), case["weights"]
    lens, t = _lens(case), _new_tokens(case)
    ids = inp["tokens"][:t] if case["path"] == "prompt" else inp["tokens"][:len(lens)]
    pos = torch.cat([torch.arange(n, n + t, device=DEVICE) for n in lens])
    pages = [torch.tensor(row, device=DEVICE) for row in inp["tables"]]
    slot = torch.cat([row[torch.arange(n, n + t, device=DEVICE) // PAGE] for row, n in zip(pages, lens)])
    x, held = inp["embed"][ids].double(), []
    for lw, pool in zip(inp["layers"], inp["pools"]):
        qkv = (_norm(x, lw["norm1"]) @ _dense(lw["qkv"], kind).t()).unflatten(1, (-1, hd))
        q, k, v = qkv[:, :hq], qkv[:, hq:hq + hkv], qkv[:, hq + hkv:]
        q, k = _rotate(q, pos, theta), _rotate(k, pos, theta)
        out = torch.empty_like(q)
        for s, n in enumerate(lens):
            at = slice(s * t, (s + 1) * t)
            out[at] = _attend(q[at], torch.cat((_rows(pool[0], pages[s], n), k[at])),
                              torch.cat((_rows(pool[1], pages[s], n), v[at])), n, case["window"])
        for (values, sb), new in zip(pool, (k, v)):
            if sb is None:
                page = values[inp["first"]:].double()
                page[slot - inp["first"], :, pos % PAGE] = new
            else:       # 8 bits per group of 64: the smallest value and the step between codes
                page, g = sb[inp["first"]:].double(), new.unflatten(-1, (-1, GROUP))
                low = g.amin(-1)
                page[slot - inp["first"], :, pos % PAGE] = torch.stack(((g.amax(-1) - low) / 255, low), -1)
            held.append(page)
        x = x + out.flatten(1) @ _dense(lw["out"], kind).t()
        h = _norm(x, lw["norm2"])
        if not experts:
            up = h @ _dense(lw["up"], kind).t()
            x = x + (torch.nn.functional.silu(up[:, :inner]) * up[:, inner:]) @ _dense(lw["down"], kind).t()
            continue
        wts, idx = torch.topk(torch.softmax(h @ lw["router"].double().t(), -1), top)
        wts, y = wts / wts.sum(-1, keepdim=True), torch.zeros_like(x)
        for e in idx.unique().tolist():
            row, col = (idx == e).nonzero(as_tuple=True)
            up = h[row] @ _dense([None if p is None else p[e] for p in lw["up"]], kind).t()
            up = torch.nn.functional.silu(up[:, :inner]) * up[:, inner:]
            y.index_add_(0, row, (up @ _dense([None if p is None else p[e] for p in lw["down"]], kind).t()) * wts[row, col, None])
        x = x + y
    if case["path"] == "prompt" and not case["all_logits"]:
        x = x[-1:]
    return {"logits": _norm(x, inp["norm"]) @ _dense(inp["head"], kind).t(), "held": held}
