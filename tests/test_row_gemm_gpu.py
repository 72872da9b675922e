"""4-bit products with W's rows as the products' rows (csrc/kernels/row_gemm.cu) against 64-bit products of the same weights, rounded to
bf16 as the kernel expands them.

Tolerances (2-norm of the difference over that of the result). fp32 results: bf16 products are exact in fp32, so what is left is the
summation, 2e-5. bf16 results add 2^-9 at most each, 3e-3. SwiGLU at these sizes about triples a relative error and is rounded once more;
its fast division adds 2^-21."""
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


def _case(dev, n, k, rows, experts=0, seed=0):
    from rmlx_b200.ops.weights import LinearWeight
    g = torch.Generator(device=dev).manual_seed(seed)
    w = LinearWeight.random(n, k, "q4", dev, experts=experts, generator=g)
    return w, w.dequantized().to(torch.bfloat16).double(), torch.randn(rows, k, device=dev, generator=g).to(torch.bfloat16), g


# one stage sequence and several, one tile of rows of W and more than one per block (n), each side of a tile's 160 rows and of the products'
# 16 and the copies' 32; K shared unevenly by the blocks of a cluster
@pytest.mark.parametrize("n,k,split", [(128, 512, 1), (384, 1536, 2), (256, 3584, 4), (128, 4096, 8), (20480, 512, 0)])
@pytest.mark.parametrize("rows", [1, 16, 33, 96, 160, 161, 330])
def test_plain(dev, n, k, split, rows):
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import row_gemm
    if rows > 96:
        split = min(split, 1)                            # the sums of more rows don't fit
    w, wd, x, g = _case(dev, n, k, rows)
    want = x.double() @ wd.t()
    got = [row_gemm(x, w, out_dtype=torch.float32, split=split) for _ in range(2)]
    GemmStatus.check(dev)
    assert _rel(got[0], want) < 2e-5 and torch.equal(got[0], got[1])
    res = torch.randn(rows, n, device=dev, generator=g).to(torch.bfloat16)
    assert _rel(row_gemm(x, w, res, split=split), want + res.double()) < 3e-3
    act = torch.nn.functional.silu(want[:, :n // 2]) * want[:, n // 2:]
    assert _rel(row_gemm(x, w, swiglu=True, split=split), act) < 3e-3
    assert _rel(row_gemm(x, w, swiglu=True, out_dtype=torch.float32, split=split), act) < 1e-4


@pytest.mark.parametrize("counts", [[3, 0, 160, 1, 161], [0, 700, 0, 0, 5], [0, 0, 0, 0, 0], [16, 17, 32, 33, 64]])
@pytest.mark.parametrize("first", [0, 40])
def test_experts(dev, counts, first):
    """Rows before the first expert's and behind the last one's belong to nobody and stay as they are."""
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import row_gemm
    rows = first + sum(counts) + 7
    w, wd, x, g = _case(dev, 256, 1024, rows, experts=len(counts), seed=1)
    offsets = (torch.tensor([0] + counts, device=dev).cumsum(0) + first).to(torch.int32)
    for swiglu in (False, True):
        out = torch.full((rows, 128 if swiglu else 256), 3.0, dtype=torch.bfloat16, device=dev)
        row_gemm(x, w, out=out, offsets=offsets, swiglu=swiglu)
        GemmStatus.check(dev)
        at = first
        for e, c in enumerate(counts):
            if c:
                want = x[at:at + c].double() @ wd[e].t()
                if swiglu:
                    want = torch.nn.functional.silu(want[:, :128]) * want[:, 128:]
                assert _rel(out[at:at + c], want) < 3e-3
            at += c
        assert (out[:first] == 3.0).all() and (out[at:] == 3.0).all()


@pytest.mark.parametrize("rows,experts", [(70, 0), (20 * 8, 8)])
def test_routes_agree(dev, rows, experts):
    """The tiles of 128 rows of x take the same bf16 weights: only the order of fp32 sums may differ."""
    from rmlx_b200.ops import quantized
    n, k = (4096, 2048) if not experts else (512, 1024)
    w, _, x, g = _case(dev, n, k, rows, experts=experts, seed=2)
    off = None if not experts else (torch.arange(experts + 1, device=dev) * (rows // experts)).to(torch.int32)
    assert quantized.row_pays(rows, n, k, experts)
    other = quantized.xgemm(x, w, offsets=off, bn=128)
    assert _rel(quantized.xgemm(x, w, offsets=off), other.double()) < 2e-3


def test_refusals(dev):
    from rmlx_b200 import _lib
    from rmlx_b200.ops.quantized import row_gemm, row_supported
    w, _, x, _ = _case(dev, 192, 512, 4)
    assert not row_supported(x, w, torch.empty(4, 192, dtype=torch.bfloat16, device=dev))
    with pytest.raises(_lib.NativeError):
        row_gemm(x, w)
    w, _, x, _ = _case(dev, 128, 512, 200)
    with pytest.raises(_lib.NativeError):
        row_gemm(x, w, split=2)                          # more than K has of 512
