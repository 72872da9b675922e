"""The router of several rows (csrc/kernels/decode_moe.cu, a cluster per eight rows) against 64-bit arithmetic."""
import pytest
import torch

from rmlx_b200.ops import decode as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e,k,top", [(128, 4096, 8), (32, 2048, 8), (256, 2056, 8), (200, 1000, 3), (16, 8, 1), (129, 40, 8), (8, 4104, 8)])
@pytest.mark.parametrize("b", [2, 8, 9, 65])
@pytest.mark.parametrize("norm", [True, False])
def test_rows(dev, e, k, top, b, norm):
    torch.manual_seed(e + k + b)
    gate = (torch.randn(e, k, device=dev) * k ** -0.5).to(torch.bfloat16)
    x = torch.randn(b, k + 8, device=dev).to(torch.bfloat16)[:, :k]                 # rows further apart than they are long
    nw = (1 + 0.1 * torch.randn(k, device=dev)).to(torch.bfloat16) if norm else None
    bias = torch.randn(e, device=dev) * 0.01
    scratch = D.RouterScratch(b, e, dev) if b > 4 else None
    counts = torch.zeros(e, dtype=torch.int32, device=dev)
    idx, wts = D.moe_router(x, gate, nw, 1e-6, top, bias, scratch, counts=counts)
    xd = x.double()
    if norm:
        xd = xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * nw.double()
    want = xd @ gate.double().t()
    # products are exact; 32 of them are added up in an instruction's adder (each at most 2^-23 off), then at most 8 + 8 + 4 fp32 sums
    # per warp step, block and cluster; the factor of the norm is four operations
    size = xd.abs() @ gate.double().abs().t()
    bound = (32 + k // 1024 + 20 + 4) * 2.0 ** -23 * size
    if scratch is not None:
        assert ((scratch.logits.double() - want).abs() <= bound).all()
    # the choices are the largest ones up to that error, and the weights their renormalised exponentials (__expf: 2 ulp and the
    # argument's rounding)
    biased = want + bias.double()
    chosen, least = biased.gather(1, idx.long()), biased.topk(top, -1).values
    slack = 2 * (bound.amax(1, keepdim=True) + 2.0 ** -22)
    assert ((chosen - least).abs() <= slack).all()
    assert all(len(set(r)) == top for r in idx.tolist())
    assert ((wts.double() - torch.softmax(chosen, -1)).abs() <= 4 * slack + 1e-5).all()
    assert torch.equal(counts.cpu().long(), torch.bincount(idx.flatten().cpu().long(), minlength=e))


def test_ties_nan_and_infinities(dev):
    """Equal logits: the lowest numbers; a row without numbers chooses none of the experts; the rows beside it are untouched."""
    gate = torch.zeros(64, 256, device=dev, dtype=torch.bfloat16)
    x = torch.ones(9, 256, device=dev, dtype=torch.bfloat16)
    idx, wts = D.moe_router(x, gate, None, 1e-6, 4)
    assert idx.tolist() == [[0, 1, 2, 3]] * 9 and torch.equal(wts, torch.full_like(wts, 0.25))
    gate[5] = 1
    x[3] = float("nan")
    x[4] = float("inf")
    idx, wts = D.moe_router(x, gate, torch.ones(256, device=dev, dtype=torch.bfloat16), 1e-6, 4)
    rows = idx.tolist()
    for r, row in enumerate(rows):
        if r in (3, 4):
            assert all(not 0 <= c < 64 for c in row)
        else:
            assert row == [5, 0, 1, 2]


def test_selection_matches_every_count(dev):
    """The selection over given logits for each number of registers that it is built for, with equal probabilities and zeros."""
    for e in (8, 32, 33, 128, 129, 256):
        empty = D.topk_route(torch.full((3, e), float("nan"), device=dev), 4)
        assert all(not 0 <= c < e for r in empty[0].tolist() for c in r) and not empty[2].any()
        logits = torch.randint(0, 4, (50, e), device=dev).float() * 30
        idx, wts, counts, offsets = D.topk_route(logits, 8)
        order = torch.sort(torch.softmax(logits, -1), dim=-1, descending=True, stable=True)
        assert torch.equal(idx.long(), order.indices[:, :8])
        w = order.values[:, :8]
        assert torch.allclose(wts, w / w.sum(-1, keepdim=True), rtol=1e-5, atol=1e-7)
        assert torch.equal(counts.cpu().long(), torch.bincount(idx.flatten().cpu().long(), minlength=e))
