"""Projections of a few rows (csrc/kernels/narrow_gemm.cu) against 64-bit products of the same weights.

Tolerances. fp32 results: codes and bf16 inputs enter the products exactly, so what is left is the fp32 summation, 2e-5 of the
result's norm. With a norm, 4-bit and 8-bit kernels round x times its weight to fp16 (2^-12 relative, independent per term):
3e-4; bf16 ones keep it in two terms. bf16 results add 2^-9."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda")


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


def _case(dev, kind, n, k, rows, experts=0, seed=0):
    from rmlx_b200.ops.weights import LinearWeight
    g = torch.Generator(device=dev).manual_seed(seed)
    w = LinearWeight.random(n, k, kind, dev, experts=experts, generator=g)
    return w, w.dequantized().double(), torch.randn(rows, k, device=dev, generator=g).to(torch.bfloat16), g


# one slab and several (K), one row tile and ragged runs of them (N), every tile count of rows and its edges
@pytest.mark.parametrize("kind", ["q4", "q8", None])
@pytest.mark.parametrize("n,k", [(16, 512), (48, 1024), (1056, 2560), (544, 4608), (64, 14336)])
@pytest.mark.parametrize("rows", [1, 8, 9, 17, 33, 64])
def test_plain(dev, kind, n, k, rows):
    from rmlx_b200.ops import narrow
    w, wd, x, g = _case(dev, kind, n, k, rows)
    assert narrow.supported(w)
    want = x.double() @ wd.t()
    for shares in (0, 1, 2, 4, 8):
        assert _rel(narrow.narrow_gemm(x, w, out_dtype=torch.float32, shares=shares), want) < 2e-5
    res = torch.randn(rows, n, device=dev, generator=g).to(torch.bfloat16)
    assert _rel(narrow.narrow_gemm(x, w, residual=res), want + res.double()) < 4e-3


@pytest.mark.parametrize("kind", ["q4", "q8", None])
@pytest.mark.parametrize("k", [512, 4096, 8192])
@pytest.mark.parametrize("rows", [1, 5, 8, 16])
def test_norm_and_swiglu(dev, kind, k, rows):
    from rmlx_b200.ops import narrow
    w, wd, x, g = _case(dev, kind, 96, k, rows, seed=1)
    nw = torch.rand(k, device=dev, generator=g).to(torch.bfloat16) + 0.5
    xd = x.double()
    up = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()) @ wd.t()
    assert _rel(narrow.narrow_gemm(x, w, nw, 1e-6, out_dtype=torch.float32), up) < (3e-4 if kind else 2e-5)
    want = torch.nn.functional.silu(up[:, :48]) * up[:, 48:]
    # a relative error e of gate and up is at most about 3 e of the activation at these sizes
    assert _rel(narrow.narrow_gemm(x, w, nw, 1e-6, out_dtype=torch.float32, swiglu=True), want) < (1e-3 if kind else 6e-5)


@pytest.mark.parametrize("kind", ["q4", "q8", None])
@pytest.mark.parametrize("rows", [1, 3, 40])
def test_expert_feed_forward(dev, kind, rows):
    """Experts without rows, with one, and with more rows than a pass holds (every row of the largest batch chooses expert 3)."""
    from rmlx_b200.ops import narrow
    e, d, inner, k = 12, 1024, 512, 4
    gu, gud, x, g = _case(dev, kind, 2 * inner, d, rows, experts=e, seed=2)
    dn, dnd, _, _ = _case(dev, kind, d, inner, 1, experts=e, seed=3)
    idx = torch.stack([torch.randperm(e - 1, device=dev, generator=g)[:k] for _ in range(rows)]).to(torch.int32)
    if rows == 40:
        idx[:, 1] = torch.where((idx == 3).any(1), idx[:, 1], torch.full_like(idx[:, 1], 3))
    wts = torch.rand(rows, k, device=dev, generator=g)
    res = torch.randn(rows, d, device=dev, generator=g).to(torch.bfloat16)
    up = torch.einsum("tsnk,tk->tsn", gud[idx.long()], x.double())
    act = torch.nn.functional.silu(up[..., :inner]) * up[..., inner:]
    y = torch.einsum("tsnk,tsk->tsn", dnd[idx.long()], act)
    want = res.double() + (y * wts.double()[..., None]).sum(1)
    # the activation is rounded to bf16 (2^-9) in between, the result at the end
    assert _rel(narrow.expert_ffn(x, idx, wts, gu, dn, residual=res), want) < 8e-3
    offsets, order = narrow.group_pairs(idx, e)
    assert torch.equal(torch.sort(order).values, torch.arange(rows * k, device=dev, dtype=torch.int32))
    flat = idx.flatten()[order.long()]
    counts = torch.bincount(flat.long(), minlength=e)
    assert torch.equal(offsets[1:].long(), counts.cumsum(0)) and bool((flat[1:] >= flat[:-1]).all())
    for tiles in (0, 1, 2, 4):
        got = narrow.narrow_gemm(x, gu, offsets=offsets, order=order, x_div=k, rows=rows * k, out_dtype=torch.float32, tiles=tiles)
        assert _rel(got, up.view(rows * k, -1)) < 2e-5


@pytest.mark.parametrize("kind", ["q4", "q8", None])
@pytest.mark.parametrize("experts,rows", [(12, 3), (256, 9)])
def test_expert_feed_forward_with_norm(dev, kind, experts, rows):
    """The form of a decode step: the norm of x inside the first projection, buffers that the caller keeps, and, at most, 256
    experts. Errors: the norm's product rounded to fp16 (4-bit, 8-bit: 3e-4), activations and the result to bf16."""
    from rmlx_b200.ops import narrow
    d, inner, k = 1024, 512, 4
    gu, gud, x, g = _case(dev, kind, 2 * inner, d, rows, experts=experts, seed=11)
    dn, dnd, _, _ = _case(dev, kind, d, inner, 1, experts=experts, seed=12)
    nw = (torch.rand(d, device=dev, generator=g) + 0.5).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(experts, device=dev, generator=g)[:k] for _ in range(rows)]).to(torch.int32)
    idx[0, 0] = experts - 1
    wts = torch.rand(rows, k, device=dev, generator=g)
    res = torch.randn(rows, d, device=dev, generator=g).to(torch.bfloat16)
    xd = x.double()
    xn = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()
    up = torch.einsum("tsnk,tk->tsn", gud[idx.long()], xn)
    act = torch.nn.functional.silu(up[..., :inner]) * up[..., inner:]
    y = torch.einsum("tsnk,tsk->tsn", dnd[idx.long()], act)
    want = res.double() + (y * wts.double()[..., None]).sum(1)
    scratch, out = narrow.ExpertScratch(rows + 3, k, gu, dn), torch.empty_like(res)
    for _ in range(2):
        assert narrow.expert_ffn(x, idx, wts, gu, dn, nw, 1e-6, residual=res, out=out, scratch=scratch) is out
        assert _rel(out, want) < 8e-3


@pytest.mark.parametrize("kind", ["q4", "q8"])
def test_extreme_inputs(dev, kind):
    """Zero groups, the smallest and largest magnitudes the activations' scaling covers, one huge value beside small ones, and
    an infinity, which stays in its own row."""
    from rmlx_b200.ops import narrow
    w, wd, x, _ = _case(dev, kind, 64, 512, 6, seed=4)
    x[0, :] = 0
    x[1, 64:128] = 0
    x[2] *= 2.0 ** -70
    x[3] *= 2.0 ** 80
    x[4, 7] = 2.0 ** 20
    want = x.double() @ wd.t()
    x[5, 3] = float("inf")
    got = narrow.narrow_gemm(x, w, out_dtype=torch.float32)
    assert float(got[0].abs().max()) == 0.0
    for r in range(1, 5):
        assert _rel(got[r], want[r]) < 2e-5
    assert not torch.isfinite(got[5]).any()


def test_refusals(dev):
    from rmlx_b200 import _lib
    from rmlx_b200.ops import narrow
    from rmlx_b200.ops.weights import LinearWeight
    for n, k in ((24, 512), (64, 320)):
        w = LinearWeight.random(n, k, "q4", dev)
        assert not narrow.supported(w)
        with pytest.raises(_lib.NativeError):
            narrow.narrow_gemm(torch.zeros(2, k, dtype=torch.bfloat16, device=dev), w)


def test_weights_that_are_views(dev):
    """A weight whose rows are not next to each other keeps the kernels that take a row stride."""
    from rmlx_b200.models.prefill import _mm
    from rmlx_b200.ops import narrow
    from rmlx_b200.ops.weights import LinearWeight, W_BF16
    g = torch.Generator(device=dev).manual_seed(5)
    wide = torch.randn(4096, 1024, device=dev, generator=g).to(torch.bfloat16)
    w = LinearWeight(W_BF16, wide[:, :512])
    assert not narrow.supported(w)
    for rows in (4, 1024):
        x = torch.randn(rows, 512, device=dev, generator=g).to(torch.bfloat16)
        assert _rel(_mm(x, w), x.double() @ w.w.double().t()) < 4e-3


@pytest.mark.parametrize("experts", [12, 256])
@pytest.mark.parametrize("bad", [-1, 0, 0x7fffffff])
def test_choices_that_are_no_expert(dev, experts, bad):
    """A slot whose choice is outside [0, E) (0 stands for E itself; a row of NaN logits gives E or the largest number) adds
    nothing and changes no other row: results are equal bit for bit to those of a batch in which it carries no weight."""
    from rmlx_b200.ops import narrow
    d, inner, rows, k = 512, 512, 5, 4
    gu, _, x, g = _case(dev, "q4", 2 * inner, d, rows, experts=experts, seed=6)
    dn, _, _, _ = _case(dev, "q4", d, inner, 1, experts=experts, seed=7)
    idx = torch.randint(0, experts, (rows, k), device=dev, generator=g).to(torch.int32)
    wts = torch.rand(rows, k, device=dev, generator=g)
    res = torch.randn(rows, d, device=dev, generator=g).to(torch.bfloat16)
    scratch = narrow.ExpertScratch(rows, k, gu, dn)
    scratch.act.fill_(float("nan")), scratch.y.fill_(float("nan"))
    none = wts.clone()
    none[1], none[3, 2] = 0.0, 0.0
    want = narrow.expert_ffn(x, idx, none, gu, dn, residual=res)
    out = idx.clone()
    out[1], out[3, 2] = bad or experts, bad or experts
    got = narrow.expert_ffn(x, out, wts, gu, dn, residual=res, scratch=scratch)
    assert torch.equal(got, want) and torch.equal(got[1], res[1])
    offsets, order = narrow.group_pairs(out, experts)
    assert int(offsets[-1]) == rows * k - k - 1
    flat = out.flatten()[order[:int(offsets[-1])].long()]
    assert torch.equal(offsets[1:].long(), torch.bincount(flat.long(), minlength=experts).cumsum(0))


@pytest.mark.parametrize("kind", ["q4", "q8"])
def test_scales_at_odd_addresses(dev, kind):
    """Several rows against weights whose scales and biases are views at an odd offset take the kernels that read those."""
    from rmlx_b200.ops import decode as D
    from rmlx_b200.ops import narrow
    from rmlx_b200.ops.weights import LinearWeight
    w, wd, x, _ = _case(dev, kind, 2048, 1024, 4, seed=8)

    def shifted(t):
        room = torch.zeros(t.numel() + 8, dtype=t.dtype, device=dev)
        return room[3:3 + t.numel()].view(t.shape).copy_(t)

    odd = LinearWeight(w.kind, w.w, shifted(w.scales), shifted(w.biases))
    assert narrow.supported(w) and not narrow.supported(odd)
    # the per-row kernels multiply in fp16 (2^-11 per product)
    assert _rel(D.rms_gemv(x, odd, out_dtype=torch.float32), x.double() @ wd.t()) < 2e-3


@pytest.mark.parametrize("kind", ["q4", "q8", None])
def test_residuals_of_another_shape(dev, kind):
    """A residual with too few rows is refused for every kind of weight; one whose rows lie apart is refused where the tensor-core
    GEMM of the same weight refuses it (bf16, 8-bit)."""
    from rmlx_b200.models.prefill import _mm
    from rmlx_b200.ops import decode as D
    from rmlx_b200.ops import narrow
    w, wd, x, g = _case(dev, kind, 2048, 1024, 6, seed=9)
    assert narrow.pays(w, 6)
    res = torch.randn(6, 2048, device=dev, generator=g).to(torch.bfloat16)
    for bad in (res[:1], res[:5], res[:, :2032].contiguous(), res.float(), res[0]):
        with pytest.raises(AssertionError):
            narrow.narrow_gemm(x, w, residual=bad)
        with pytest.raises(AssertionError):
            D.rms_gemv(x, w, residual=bad)
    wide = torch.zeros(6, 2056, dtype=torch.bfloat16, device=dev)
    wide[:, :2048] = res
    if kind != "q4":
        for bad in (res[:1], wide[:, :2048]):
            with pytest.raises(AssertionError):
                _mm(x, w, residual=bad)
    want = x.double() @ wd.t() + res.double()
    assert _rel(_mm(x, w, residual=res), want) < 4e-3
    assert _rel(narrow.narrow_gemm(x, w, residual=wide[:, :2048]), want) < 4e-3


@pytest.mark.parametrize("k", [2048, 14336])
@pytest.mark.parametrize("norm", [False, True])
def test_sums_of_bf16_weights(dev, k, norm):
    """Products of bf16 are exact in fp32, so the error is that of adding them up: K / 64 rounded additions of 2^-24 each (in a
    random walk 4e-7 for the longest K), and what the tensor cores cut inside 64 of K. With one sum in the tensor cores it is 2e-6."""
    from rmlx_b200.ops import narrow
    w, wd, x, g = _case(dev, None, 512, k, 5, seed=10)
    nw = (torch.rand(k, device=dev, generator=g) + 0.5).to(torch.bfloat16) if norm else None
    xd = x.double()
    want = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double() if norm else xd) @ wd.t()
    for shares in (0, 1):
        assert _rel(narrow.narrow_gemm(x, w, nw, 1e-6, out_dtype=torch.float32, shares=shares), want) < 5e-7


@pytest.mark.parametrize("rows", [2, 3, 4])
@pytest.mark.parametrize("n,k,norm", [(1024, 2048, True), (1024, 4096, True), (1024, 8192, False), (512, 9216, False), (640, 15424, False)])
def test_bf16_rows_on_either_side_of_the_rule(dev, rows, n, k, norm):
    """Two and three rows of bf16 weights stay on the per-row kernels where those stream as fast: both add in fp32, so the error does
    not tell which one ran (random walk of K / 64 additions; the per-row kernels add K / 32 per lane and the lanes in a tree)."""
    from rmlx_b200.ops import decode as D
    w, wd, x, g = _case(dev, None, n, k, rows, seed=13)
    nw = (torch.rand(k, device=dev, generator=g) + 0.5).to(torch.bfloat16) if norm else None
    xd = x.double()
    want = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double() if norm else xd) @ wd.t()
    assert D._several(rows, w, x, nw) == (rows == 4 or rows * k > 30720 or (rows == 2 and not (k > (2048 if norm else 8192))) or rows == 3)
    assert _rel(D.rms_gemv(x, w, nw, 1e-6, out_dtype=torch.float32), want) < 1e-6


# the even split: clusters of which every block takes a ragged share of K, more tiles per cluster than fit its sums at once
#, rows of W beyond what a cluster's buffers hold, experts on clusters
@pytest.mark.parametrize("kind,n,k,rows,shares", [("q4", 80, 2560, 16, 4), ("q8", 208, 3584, 11, 2), ("q4", 72000, 4096, 16, 2),
                                                  ("q8", 64, 33280, 3, 0), ("q4", 32, 32768, 12, 0)])
def test_clusters(dev, kind, n, k, rows, shares):
    from rmlx_b200.ops import narrow
    w, _, x, g = _case(dev, kind, min(n, 8000), k, rows, seed=7)
    if n > 8000:                                         # the reference of 8000 rows nine times over
        w = type(w)(w.kind, *(t.repeat(n // 8000, 1) for t in (w.w, w.scales, w.biases)))
    want = (x.double() @ w.dequantized()[:8000].double().t()).repeat(1, max(1, n // 8000))
    got = [narrow.narrow_gemm(x, w, out_dtype=torch.float32, shares=shares) for _ in range(3)]
    assert _rel(got[0], want) < 2e-5 and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("kind", ["q4", "q8"])
@pytest.mark.parametrize("k,tiles,shares", [(8192, 1, 0), (3072, 2, 2), (512, 1, 1)])
def test_experts_on_clusters(dev, kind, k, tiles, shares):
    """No rows, one row and several passes of rows per expert."""
    from rmlx_b200.ops import narrow
    counts = [0, 1, 8, 0, 19, 3, 33, 0]
    rows = sum(counts)
    w, wd, x, g = _case(dev, kind, 112, k, rows, experts=len(counts), seed=8)
    offsets = torch.tensor([0] + counts, device=dev).cumsum(0).to(torch.int32)
    order = torch.randperm(rows, device=dev, generator=g).to(torch.int32)
    got = narrow.narrow_gemm(x, w, out_dtype=torch.float32, offsets=offsets, order=order, rows=rows, tiles=tiles, shares=shares)
    at = 0
    for e, c in enumerate(counts):
        r = order[at:at + c].long()
        at += c
        if c:
            assert _rel(got[r], x[r].double() @ wd[e].t()) < 2e-5


@pytest.mark.parametrize("rows,top,experts", [(1, 8, 128), (5, 3, 7), (64, 8, 128), (129, 8, 256), (192, 8, 32), (700, 2, 16)])
def test_pairs_in_order(dev, rows, top, experts):
    """The pairs of an expert in ascending order, each once, without those that chose none: a pair's place decides how its sums are
    split, so results would otherwise differ from run to run."""
    from rmlx_b200.ops import narrow
    g = torch.Generator(device=dev).manual_seed(rows)
    idx = torch.randint(-1, experts + 1, (rows, top), device=dev, generator=g, dtype=torch.int32)
    offsets, order = narrow.group_pairs(idx, experts)
    flat = idx.flatten().tolist()
    lists = [[i for i, e in enumerate(flat) if e == x] for x in range(experts)]
    assert offsets.tolist() == [sum(len(p) for p in lists[:x]) for x in range(experts + 1)]
    assert order[:sum(map(len, lists))].tolist() == [i for p in lists for i in p]


@pytest.mark.parametrize("kind,n,k,wide", [("q4", 16384, 2048, True), ("q8", 16400, 2048, True), ("q4", 16384, 1536, False), ("q8", 8192, 4096, False),
                                           (None, 16384, 2048, False)])
def test_one_row_of_a_wide_weight(dev, kind, n, k, wide):
    from rmlx_b200.ops import decode as D
    w, wd, x, g = _case(dev, kind, n, k, 1, seed=17)
    res = torch.randn(1, n, device=dev, generator=g).to(torch.bfloat16)
    assert D._several(1, w, x) == wide and D._several(1, w, x, swiglu=True) is False
    # the weight-streaming kernel's sums are fp32; the per-row kernels multiply 4- and 8-bit weights in fp16
    bound = 1e-5 if wide or kind is None else 2e-3
    assert _rel(D.rms_gemv(x, w, residual=res, out_dtype=torch.float32), x.double() @ wd.t() + res.double()) < bound


@pytest.mark.parametrize("kind", ["q4", "q8"])
@pytest.mark.parametrize("rows,top,experts,k,n", [(1, 8, 128, 512, 32), (1, 1, 2, 1536, 96), (4, 8, 16, 1024, 64), (3, 5, 7, 4096, 160), (1, 32, 40, 8192, 32)])
def test_pairs(dev, kind, rows, top, experts, k, n):
    """Pairs one by one: every expert's rows, choices that are no expert, an expert chosen twice, norm, SwiGLU; then down and combined."""
    from rmlx_b200.ops import narrow
    w, wd, x, g = _case(dev, kind, n, k, rows, experts=experts, seed=19)
    nw = (torch.rand(k, device=dev, generator=g) + 0.5).to(torch.bfloat16)
    idx = torch.randint(0, experts, (rows, top), device=dev, generator=g, dtype=torch.int32)
    if rows * top > 1:
        idx[0, 0] = experts
        idx[-1, -1] = 0x7fffffff
    flat = idx.flatten().tolist()
    real = [i for i, e in enumerate(flat) if e < experts]
    xd = x.double()
    xn = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()
    for norm, src in ((None, xd), (nw, xn)):
        out = torch.full((rows * top, n), 7.0, device=dev)
        narrow.pairs_gemm(x, w, idx, top, out, norm)
        want = torch.stack([src[i // top] @ wd[flat[i]].t() for i in real])
        # without a norm x is exact in the products; with one it is rounded to fp16, 2^-12 of each value at most, half that on average
        assert _rel(out[real], want) < (2e-5 if norm is None else 2.0 ** -11)
        assert all(bool((out[i] == 7.0).all()) for i in range(rows * top) if i not in real)
    act = torch.zeros(rows * top, n // 2, device=dev, dtype=torch.bfloat16)
    narrow.pairs_gemm(x, w, idx, top, act, nw, swiglu=True)
    gate, up = want[:, :n // 2], want[:, n // 2:]
    assert _rel(act[real], gate * torch.sigmoid(gate) * up) < 6e-3
    # a row of its own for each pair
    y = torch.randn(rows * top, k, device=dev, generator=g).to(torch.bfloat16)
    out = torch.zeros(rows * top, n, device=dev)
    narrow.pairs_gemm(y, w, idx, 1, out)
    assert _rel(out[real], torch.stack([y[i].double() @ wd[flat[i]].t() for i in real])) < 2e-5


def test_pairs_in_a_decode_step(dev):
    """Steps of 1 to 4 rows whose experts go pair by pair against the streaming kernels: the same tokens' logits within the latter's
    rounding (they multiply in fp16, 1e-3 a projection)."""
    from rmlx_b200.ops import decode as D, narrow
    from rmlx_b200.ops.weights import LinearWeight
    g = torch.Generator(device=dev).manual_seed(3)
    up, down = (LinearWeight.random(a, b, "q4", dev, experts=16, generator=g) for a, b in ((28672, 2048), (2048, 14336)))
    assert [narrow.pays_pairs(up, down, r, 2) for r in (0, 1, 2, 4, 9, 17)] == [False, True, True, True, False, False] and D.pairs_apart()
    x = torch.randn(4, 2048, device=dev, generator=g).to(torch.bfloat16)
    nw = torch.ones(2048, device=dev, dtype=torch.bfloat16)
    sc = narrow.ExpertScratch(4, 2, up, down)
    for r in (1, 4):
        idx = torch.stack([torch.randperm(16, device=dev, generator=g)[:2] for _ in range(r)]).int().contiguous()
        wts = torch.rand(r, 2, device=dev, generator=g)
        got = narrow.pairs_ffn(x[:r], idx, wts, up, down, nw, 1e-6, x[:r], torch.empty_like(x[:r]), sc)
        act = D.moe_gate_up(x[:r], up, nw, 1e-6, idx)
        want = D.moe_down(act, down, idx, wts, residual=x[:r])
        assert _rel(got.float() - x[:r].float(), (want.float() - x[:r].float()).double()) < 1e-2


@pytest.mark.parametrize("kind,rows", [("q4", 1), ("q4", 3), ("q8", 2)])
def test_experts_narrower_than_the_scratch(dev, kind, rows):
    """A scratch made for wider experts gives the same results to the bit as one of the experts' own width."""
    from rmlx_b200.ops import narrow
    from rmlx_b200.ops.weights import LinearWeight
    g = torch.Generator(device=dev).manual_seed(4)
    d, top, experts = 1024, 4, 16
    wide, own = (tuple(LinearWeight.random(a, b, kind, dev, experts=experts, generator=g) for a, b in ((2 * inner, d), (d, inner)))
                 for inner in (1536, 512))
    x = torch.randn(rows, d, device=dev, generator=g).to(torch.bfloat16)
    nw = torch.ones(d, device=dev, dtype=torch.bfloat16)
    idx = torch.randint(0, experts, (rows, top), device=dev, generator=g, dtype=torch.int32)
    wts = torch.rand(rows, top, device=dev, generator=g)
    for ffn in (narrow.expert_ffn, narrow.pairs_ffn):
        got, want = (ffn(x, idx, wts, *own, nw, 1e-6, residual=x, out=torch.empty_like(x), scratch=narrow.ExpertScratch(rows, top, *of))
                     for of in (wide, own))
        assert torch.equal(got, want)
