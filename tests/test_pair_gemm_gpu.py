"""The tensor-core GEMM on SM pairs (csrc/kernels/pair_gemm.cu): the same products in the same order as the single-SM tiles, so
plain results are equal bit for bit; against 64 bits the error is that of a bf16 result (and, for 4-bit weights, of weights
rounded to bf16).

Bounds: a rounding to bf16 is off by at most 2^-9 = 1.96e-3 of the value, so a result of bf16 weights by at most that of its norm
(ROUND, with room for the fp32 sums); weights rounded to bf16 add at most as much again before anything averages out, and a
gated activation, gate and up rounded each, at most three times that."""
import pytest
import torch

ROUND = 2.0e-3

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda")


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


def _case(dev, kind, m, n, k, experts=0, seed=0):
    from rmlx_b200.ops.weights import LinearWeight
    g = torch.Generator(device=dev).manual_seed(seed)
    w = LinearWeight.random(n, k, kind, dev, experts=experts, generator=g)
    return w, w.dequantized().double(), torch.randn(m, k, device=dev, generator=g).to(torch.bfloat16), g


# one row, half a pair's rows and one more, more tiles than pairs, columns that end inside a tile
@pytest.mark.parametrize("kind", [None, "q4"])
@pytest.mark.parametrize("m,n,k", [(1, 256, 512), (129, 288, 1024), (256, 256, 4096), (300, 544, 1536), (2600, 2048, 512)])
def test_plain(dev, kind, m, n, k):
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import pair_gemm, xgemm
    w, wd, x, g = _case(dev, kind, m, n, k)
    want = x.double() @ wd.t()
    got = pair_gemm(x, w)
    assert torch.equal(got, xgemm(x, w, bn=128))
    assert _rel(got, want) < (2 * ROUND if kind else ROUND)
    res = torch.randn(m, n, device=dev, generator=g).to(torch.bfloat16)
    assert _rel(pair_gemm(x, w, residual=res), want + res.double()) < 2 * ROUND
    if n % 256 == 0:
        act = torch.nn.functional.silu(want[:, :n // 2]) * want[:, n // 2:]
        assert _rel(pair_gemm(x, w, swiglu=True), act) < (4 * ROUND if kind else ROUND)
    GemmStatus.check(dev)


@pytest.mark.parametrize("kind", [None, "q4"])
@pytest.mark.parametrize("k", [512, 520, 1000, 4096])
def test_many_runs_and_tiles(dev, kind, k):
    """More tiles than pairs of SMs (162 for 74), K that ends inside a block of 64 (bf16), run after run: bit for bit the
    single-SM tiles. The blocks of a pair rely on each other's signals (see the kernel); a signal that came too early would show."""
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import pair_gemm, xgemm
    if kind and k % 512:
        pytest.skip("4-bit weights come 512 of K at a time")
    w, wd, x, g = _case(dev, kind, 2304, 4608, k, seed=5)
    want, act = xgemm(x, w, bn=128), xgemm(x, w, bn=128, swiglu=True)
    assert _rel(want, x.double() @ wd.t()) < (2 * ROUND if kind else ROUND)
    out, half = torch.empty_like(want), torch.empty_like(act)
    for _ in range(60):
        out.zero_(), half.zero_()
        assert torch.equal(pair_gemm(x, w, out=out), want)
        assert torch.equal(pair_gemm(x, w, out=half, swiglu=True), act)
    GemmStatus.check(dev)


@pytest.mark.parametrize("kind", [None, "q4"])
@pytest.mark.parametrize("m,n,k", [(40, 256, 512), (300, 544, 1024), (700, 512, 2048)])
def test_stacked_tiles(dev, kind, m, n, k):
    """``bn=-128``, two row blocks per staged block of W, against the tiles of 128 columns: plain, residual, SwiGLU, grouped."""
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import xgemm
    w, _, x, g = _case(dev, kind, m, n, k, seed=6)
    res = torch.randn(m, n, device=dev, generator=g).to(torch.bfloat16)
    assert torch.equal(xgemm(x, w, bn=-128), xgemm(x, w, bn=128))
    assert torch.equal(xgemm(x, w, residual=res, bn=-128), xgemm(x, w, residual=res, bn=128))
    if n % 256 == 0:
        assert torch.equal(xgemm(x, w, bn=-128, swiglu=True), xgemm(x, w, bn=128, swiglu=True))
        counts = [m // 2, 0, 1, m - m // 2 - 1]
        we, _, _, _ = _case(dev, kind, 1, n, k, experts=4, seed=7)
        off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=dev)
        for swiglu in (False, True):
            assert torch.equal(xgemm(x, we, offsets=off, bn=-128, swiglu=swiglu), xgemm(x, we, offsets=off, bn=128, swiglu=swiglu))
    GemmStatus.check(dev)


@pytest.mark.parametrize("kind", [None, "q4"])
def test_grouped(dev, kind):
    """Experts without rows, with one, with a whole tile and with more."""
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import pair_gemm
    counts = [3, 0, 300, 256, 1, 130]
    w, wd, x, _ = _case(dev, kind, sum(counts), 512, 1024, experts=len(counts), seed=1)
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=dev)
    want = torch.cat([x[off[e]:off[e + 1]].double() @ wd[e].t() for e in range(len(counts))])
    assert _rel(pair_gemm(x, w, offsets=off), want) < (2 * ROUND if kind else ROUND)
    act = torch.nn.functional.silu(want[:, :256]) * want[:, 256:]
    assert _rel(pair_gemm(x, w, offsets=off, swiglu=True), act) < (4 * ROUND if kind else ROUND)
    GemmStatus.check(dev)


@pytest.mark.parametrize("kind", [None, "q4"])
@pytest.mark.parametrize("m", [128, 129, 700, 2048])
def test_rule_changes_no_result(dev, kind, m):
    """``xgemm`` on either side of the rule, with rows of x apart and results that are views, 16-byte aligned (SM pairs) and not
    (single SMs, stored element by element): the same values, and nothing beside them is written."""
    from rmlx_b200.ops.quantized import pair_pays, xgemm
    w, _, x, g = _case(dev, kind, m, 4096, 512, seed=2)
    assert pair_pays(w.kind, 2048, 4096, 512) and not pair_pays(w.kind, 128, 4096, 512)
    res = torch.randn(m, 4096, device=dev, generator=g).to(torch.bfloat16)
    want, more, act = xgemm(x, w, bn=128), xgemm(x, w, residual=res, bn=128), xgemm(x, w, bn=128, swiglu=True)
    assert torch.equal(xgemm(x, w), want)
    for stride, at in ((4104, 0), (4104, 8), (4100, 0), (4104, 1), (4101, 3)):
        room = torch.zeros(m * stride + 8, dtype=torch.bfloat16, device=dev)
        wide = torch.zeros(m * stride + 8, dtype=torch.bfloat16, device=dev)
        out = room[at:at + m * stride].view(m, stride)[:, :4096]
        r = wide[at:at + m * stride].view(m, stride)[:, :4096]
        r.copy_(res)
        assert torch.equal(xgemm(x, w, out=out), want)
        assert torch.equal(xgemm(x, w, residual=r, out=out), more)
        out.zero_()
        assert torch.equal(xgemm(x, w, out=out[:, :2048], swiglu=True), act)
        out[:, :2048].zero_()
        assert not bool(room.any())
    x2 = torch.zeros(m, 520, dtype=torch.bfloat16, device=dev)
    x2[:, :512] = x
    assert torch.equal(xgemm(x2[:, :512], w), want)


@pytest.mark.parametrize("kind", [None, "q4"])
@pytest.mark.parametrize("n", [33, 100, 1001])
def test_any_number_of_columns(dev, kind, n):
    """Rows of a result of any number of columns start at any address: more than one piece of 32 columns, ends inside a piece."""
    from rmlx_b200.ops.quantized import xgemm
    w, wd, x, _ = _case(dev, kind, 150, n, 512, seed=4)
    assert _rel(xgemm(x, w), x.double() @ wd.t()) < (2 * ROUND if kind else ROUND)


@pytest.mark.parametrize("kind", [None, "q4"])
def test_residual_with_more_rows(dev, kind):
    """``xgemm`` takes the first rows of a longer residual on either side of the rule, and refuses one that is too short or has
    another row stride."""
    from rmlx_b200.ops.quantized import pair_pays, xgemm
    w, _, x, g = _case(dev, kind, 2048, 4096, 512, seed=3)
    assert pair_pays(w.kind, 2048, 4096, 512)
    res = torch.randn(2050, 4096, device=dev, generator=g).to(torch.bfloat16)
    for m in (100, 2048):
        assert torch.equal(xgemm(x[:m], w, residual=res), xgemm(x[:m], w, residual=res[:m]))
        wide = torch.zeros(m, 4104, dtype=torch.bfloat16, device=dev)
        for bad in (res[:m - 1], wide[:, :4096]):
            with pytest.raises(AssertionError):
                xgemm(x[:m], w, residual=bad)
