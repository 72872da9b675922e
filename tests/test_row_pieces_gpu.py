"""The small row kernels in 16-byte pieces (norm, rotation and cache append, page expansion, arg-max) at the edges of their pieces, and
beside tables at odd addresses, which go one value at a time."""
import pytest
import torch

from rmlx_b200.ops import decode as D

pytestmark = pytest.mark.gpu


def _at(t, odd):
    """A copy of t that starts ``odd`` elements into its storage."""
    buf = torch.empty(t.numel() + odd, dtype=t.dtype, device=t.device)
    out = buf[odd:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("d", [8, 264, 2048, 2056, 4104, 8192, 8200, 1001])
@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("weight", [True, False])
def test_rms_norm(dev, d, odd, weight):
    torch.manual_seed(d)
    x, r = (_at(torch.randn(5, d, device=dev).to(torch.bfloat16), odd) for _ in range(2))
    w = (1 + 0.1 * torch.randn(d, device=dev)).to(torch.bfloat16) if weight else None
    for res, total in ((None, False), (r, True), (r, False)):
        s = torch.empty_like(x) if total else None
        got = D.rms_norm(x, w, 1e-6, residual=res, sum_out=s) if total else D.rms_norm(x, w, 1e-6, residual=res)
        v = x if res is None else (x.float() + res.float()).to(torch.bfloat16)
        vd = v.double()
        want = vd * torch.rsqrt(vd.square().mean(-1, keepdim=True) + 1e-6) * (1 if w is None else w.double())
        # one rounding to bf16 (2^-8 at its largest) and fp32 before it
        assert ((got.double() - want).abs() <= want.abs() * (2.0 ** -8 + 1e-5) + 1e-30).all()
        assert s is None or torch.equal(s, v)


@pytest.mark.parametrize("hd,q8", [(16, False), (48, False), (64, False), (128, False), (256, False), (20, False), (64, True), (128, True), (256, True)])
@pytest.mark.parametrize("tokens,fp32", [(1, True), (7, False), (130, False)])
@pytest.mark.parametrize("traditional", [False, True])
@pytest.mark.parametrize("odd", [0, 1])
def test_rope_and_append(dev, hd, q8, tokens, fp32, traditional, odd):
    torch.manual_seed(hd + tokens)
    hq, hkv, page = 9, 2, 16
    fp32 = fp32 and not q8
    qkv = _at(torch.randn(tokens, (hq + 2 * hkv) * hd, device=dev).to(torch.float32 if fp32 else torch.bfloat16), odd)
    pos = torch.arange(5, 5 + tokens, dtype=torch.int32, device=dev)
    ang = torch.randn(5 + tokens, hd // 2, device=dev)
    cos, sin = ang.cos(), ang.sin()
    blocks = (tokens + 5) // page + 2
    table = torch.randperm(blocks, device=dev).to(torch.int32).view(1, -1)
    seq = torch.zeros(tokens, dtype=torch.int32, device=dev)
    q = torch.zeros(tokens, hq, hd, dtype=torch.bfloat16, device=dev)
    kc, vc = (torch.zeros(blocks, hkv, page, hd, dtype=torch.uint8 if q8 else torch.bfloat16, device=dev) for _ in range(2))
    sb = {n: torch.zeros(blocks, hkv, page, hd // 64, 2, dtype=torch.bfloat16, device=dev) for n in ("k_sb", "v_sb")} if q8 else {}
    D.rope_kv_write(qkv, q, kc, vc, table, pos, cos, sin, hq, hkv, token_seq=seq, traditional=traditional, **sb)
    x = qkv.double().view(tokens, hq + 2 * hkv, hd)
    c, s = (t[pos.long()].double().view(tokens, 1, -1) for t in (cos, sin))
    rot = x.clone()
    a, b = (x[..., 0::2], x[..., 1::2]) if traditional else (x[..., :hd // 2], x[..., hd // 2:])
    if traditional:
        rot[..., 0::2], rot[..., 1::2] = a * c - b * s, b * c + a * s
    else:
        rot[..., :hd // 2], rot[..., hd // 2:] = a * c - b * s, b * c + a * s
    size = x.abs().amax()
    near = lambda got, want, tol: ((got.double() - want).abs() <= tol).all()
    assert near(q, rot[:, :hq], rot[:, :hq].abs() * 2.0 ** -8 + size * 1e-6)
    where = table[0, (pos // page).long()].long()
    for cache, n, want in ((kc, "k_sb", rot[:, hq:hq + hkv]), (vc, "v_sb", x[:, hq + hkv:])):
        got = cache[where, :, (pos % page).long()]
        if q8:                                           # half a step of 1/255 of a group's range, both rounded outwards to bf16
            row = torch.arange(blocks, dtype=torch.int32, device=dev)
            full = D.kv_dequant_pages(cache, sb[n], row, blocks)
            off = D.kv_dequant_pages(_at(cache, 1), sb[n], row, blocks)
            assert torch.equal(full, off)
            got = full[where, :, (pos % page).long()]
            g = want.reshape(tokens, hkv, hd // 64, 64)
            step = (g.amax(-1) - g.amin(-1) + g.abs().amax(-1) * 2.0 ** -7) / 255 * (1 + 2.0 ** -7)
            tol = (step.unsqueeze(-1) * 0.51).expand_as(g).reshape(want.shape) + want.abs() * 2.0 ** -8
        else:
            tol = want.abs() * 2.0 ** -8 + size * 1e-6
        assert near(got, want, tol)


@pytest.mark.parametrize("rows,v,odd", [(1, 3, 0), (64, 151936, 0), (70, 4097, 0), (200, 5003, 1), (3, 32768, 1), (300, 8192, 0)])
def test_argmax(dev, rows, v, odd):
    torch.manual_seed(v)
    logits = _at(torch.randint(0, 50, (rows, v), device=dev).float(), odd)          # many equal ones: the lowest index
    logits[0] = float("-inf")
    logits[0, v - 1] = -3.0                              # the last value of a row
    if rows > 1:
        logits[1] = float("nan")
        logits[1, v // 2] = 7.0
    got = D.argmax(logits).tolist()
    clean = torch.where(logits.isnan(), torch.full_like(logits, float("-inf")), logits).cpu()
    assert got == [int((r == r.max()).nonzero()[0]) for r in clean]


@pytest.mark.parametrize("rows,v", [(1, 2044), (1, 2048), (2, 2052), (74, 20000), (75, 20000), (148, 9001), (149, 12288)])
def test_argmax_slices(dev, rows, v):
    """Short rows, and rows in as many slices as there are SMs for each."""
    torch.manual_seed(v)
    logits = torch.randint(0, 200, (rows, v), device=dev).float()
    assert D.argmax(logits).tolist() == [int((r == r.max()).nonzero()[0]) for r in logits.cpu()]


@pytest.mark.parametrize("hq,hkv,hd", [(1, 1, 64), (1, 1, 512), (26, 3, 128), (27, 3, 128), (60, 4, 128)])
def test_rotation_of_few_and_many_heads(dev, hq, hkv, hd):
    """130 tokens in pieces, by blocks as wide as their heads need, against the same tokens in two halves, one pair at a time; both round
    once to bf16."""
    torch.manual_seed(hd + hq)
    tokens, page, heads = 130, 16, hq + 2 * hkv
    qkv = torch.randn(tokens, heads * hd, device=dev).to(torch.bfloat16)
    pos = torch.arange(tokens, dtype=torch.int32, device=dev)
    ang = torch.randn(tokens, hd // 2, device=dev)
    table = torch.arange(9, dtype=torch.int32, device=dev).view(1, -1)
    res = []
    for parts in ((slice(0, 130),), (slice(0, 65), slice(65, 130))):
        q = torch.zeros(tokens, hq, hd, dtype=torch.bfloat16, device=dev)
        kc, vc = (torch.zeros(9, hkv, page, hd, dtype=torch.bfloat16, device=dev) for _ in range(2))
        for s in parts:
            D.rope_kv_write(qkv[s], q[s], kc, vc, table, pos[s], ang.cos(), ang.sin(), hq, hkv, token_seq=torch.zeros_like(pos[s]))
        res.append((q, kc, vc))
    size = float(qkv.abs().max())
    for a, b in zip(*res):
        assert ((a.double() - b.double()).abs() <= b.double().abs() * 2.0 ** -7 + size * 1e-6).all()
    assert torch.equal(res[0][2], res[1][2]) and res[0][0].any()
