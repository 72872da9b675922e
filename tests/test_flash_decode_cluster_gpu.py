"""Decode attention on clusters (csrc/kernels/flash_decode_cluster.cu) against 64-bit attention over the same cache values.

Tolerances (2-norm of the difference over that of the result). The result is rounded to bf16, 2^-9 at most and 1.7e-3 on average. bf16
cache: probabilities enter as bf16 too, independent errors of 2^-9 at most each: 3e-3 together. 8-bit cache: probabilities times scales keep
11 bits: 2e-3. A window of one key returns that key."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda")


def _cache(dev, g, lens, hkv, hd, q8):
    """(k, v, k_sb, v_sb), their values in fp64, the block table (pages shuffled) and the lengths."""
    need = [max(1, -(-n // 16)) for n in lens]
    pages = sum(need) + 1
    perm = (torch.randperm(pages - 1, device=dev, generator=g) + 1).int()
    table, at = torch.zeros(len(lens), max(need) + 3, dtype=torch.int32, device=dev), 0
    for i, n in enumerate(need):
        table[i, :n] = perm[at:at + n]
        at += n
    out, vals = [], []
    for _ in range(2):
        if q8:
            codes = torch.randint(0, 256, (pages, hkv, 16, hd), dtype=torch.uint8, device=dev, generator=g)
            # scales of very different sizes from page to page: the accumulators follow the largest so far
            s = torch.empty(pages, hkv, 16, hd // 64, device=dev).uniform_(0.75, 1.25, generator=g) * 0.0136
            s = (s * torch.randint(0, 5, (pages, 1, 1, 1), device=dev, generator=g).float().exp2() / 4).to(torch.bfloat16)
            b = (-127.5 * s.float()).to(torch.bfloat16)
            vals.append((codes.double().unflatten(-1, (-1, 64)) * s.double()[..., None] + b.double()[..., None]).flatten(-2))
            out.append((codes, torch.stack([s, b], -1).contiguous()))
        else:
            x = torch.randn(pages, hkv, 16, hd, device=dev, generator=g).to(torch.bfloat16)
            vals.append(x.double())
            out.append((x, None))
    return (out[0][0], out[1][0], out[0][1], out[1][1]), vals, table, torch.tensor(lens, dtype=torch.int32, device=dev)


def _want(q, vals, table, lens, window):
    b, hq, hd = q.shape
    hkv = vals[0].shape[1]
    out = torch.zeros(b, hq, hd, dtype=torch.double, device=q.device)
    for i, n in enumerate(lens):
        first = max(0, n - window) if window else 0
        if n:
            k, v = (x[table[i, :-(-n // 16)].long()].transpose(1, 2).flatten(0, 1)[first:n] for x in vals)
            s = torch.einsum("hgd,nhd->hgn", q[i].double().unflatten(0, (hkv, -1)), k) / math.sqrt(hd)
            out[i] = torch.einsum("hgn,nhd->hgd", torch.softmax(s, -1), v).flatten(0, 1)
    return out


# one tile on a whole cluster; short and empty sequences; more tiles than clusters (lengths far apart: the runs of tiles follow the pages);
# sixteen, fewer and more query heads per kv head than a tile has
@pytest.mark.parametrize("q8", [False, True])
@pytest.mark.parametrize("hq,hkv,hd,lens", [
    (16, 1, 128, [4097]), (4, 2, 64, [25]), (40, 2, 64, [0, 1, 16, 17, 300]), (32, 8, 128, [900, 3, 44, 2000]),
    (8, 8, 128, [37] * 90 + [1500]), (64, 4, 128, [15 + 61 * (i % 7) for i in range(80)])])
@pytest.mark.parametrize("window", [0, 33])
def test_against_exact(dev, q8, hq, hkv, hd, lens, window):
    from rmlx_b200.ops import decode as D
    g = torch.Generator(device=dev).manual_seed(len(lens) + hd)
    (k, v, ks, vs), vals, table, sl = _cache(dev, g, lens, hkv, hd, q8)
    q = torch.randn(len(lens), hq, hd, device=dev, generator=g).to(torch.bfloat16)
    want = _want(q, vals, table, lens, window)
    for longest in (max(lens), 8192):                    # other plans
        sc = D.FlashDecodeScratch(len(lens), hq, hkv, hd, 2, dev, max_len=longest)
        assert sc.clusters and sc.clusters_q8
        got = [D.flash_decode_paged(q, k, v, table, sl, None, None, sc, window, k_sb=ks, v_sb=vs) for _ in range(2)]
        assert torch.equal(got[0], got[1])
        assert float((got[0].double() - want).norm() / want.norm()) < (2e-3 if q8 else 3e-3)
        for i, n in enumerate(lens):
            if n == 0:
                assert not got[0][i].any()


@pytest.mark.parametrize("q8", [False, True])
def test_settled_cache(dev, q8):
    """Chained launches that append a token and attend to it, with pages asked for before the append has finished."""
    from rmlx_b200.ops import decode as D
    hq, hkv, hd, lens = 16, 4, 128, [1, 16, 17, 500, 2047]
    g = torch.Generator(device=dev).manual_seed(3)
    (k, v, ks, vs), _, table, sl = _cache(dev, g, lens, hkv, hd, q8)
    sc = D.FlashDecodeScratch(len(lens), hq, hkv, hd, 2, dev, max_len=2048)
    cos = torch.ones(2048, hd // 2, device=dev)
    sin = torch.zeros_like(cos)
    pos, sb = sl - 1, dict(k_sb=ks, v_sb=vs) if q8 else {}
    outs = []
    for pdl in (False, True):
        got = []
        for i in range(20):
            qkv = torch.randn(len(lens), (hq + 2 * hkv) * hd, device=dev, generator=torch.Generator(device=dev).manual_seed(i)).to(torch.bfloat16)
            q = torch.empty(len(lens), hq, hd, dtype=torch.bfloat16, device=dev)
            D.rope_kv_write(qkv, q, k, v, table, pos, cos, sin, hq, hkv, pdl=pdl, **sb)
            got.append(D.flash_decode_paged(q, k, v, table, sl, None, None, sc, pdl=pdl, settled=pdl, **sb))
        outs.append(torch.stack(got))
    assert torch.equal(outs[0], outs[1])


def test_cluster_sizes(dev):
    """One block per tile from one tile per SM on and for few pages; several where few tiles have many."""
    from rmlx_b200.ops import decode as D
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    for batch, hq, hkv, max_len, q8, one in [(sms // 4, 64, 4, 8192, False, True), (sms, 8, 1, 8192, True, True), (48, 32, 8, 8192, False, True),
                                             (1, 64, 4, 255, False, False), (1, 64, 4, 240, False, True), (2, 64, 4, 100, True, True),
                                             (1, 64, 4, 8192, False, False), (16, 32, 8, 8192, True, False)]:
        assert (D.cluster_plan(batch, hq, hkv, 128, max_len, q8) >> 16 == 1) is one


@pytest.mark.parametrize("hkv,lens", [(8, [37] * 90 + [1500]), (4, [15 + 61 * (i % 7) for i in range(150)])])
def test_runs_of_tiles_bf16(dev, hkv, lens):
    """More tiles than clusters in a bf16 cache, lengths far apart, whichever kernel the rule prefers there."""
    from rmlx_b200.ops import decode as D
    g = torch.Generator(device=dev).manual_seed(5)
    (k, v, _, _), vals, table, sl = _cache(dev, g, lens, hkv, 128, False)
    q = torch.randn(len(lens), 4 * hkv, 128, device=dev, generator=g).to(torch.bfloat16)
    want = _want(q, vals, table, lens, 0)
    sc = D.FlashDecodeScratch(len(lens), 4 * hkv, hkv, 128, 1, dev, max_len=max(lens))
    real, got = D.clusters_pay, []
    for use in (True, False):
        D.clusters_pay = lambda *a: use
        try:
            got.append(D.flash_decode_paged(q, k, v, table, sl, scratch=sc))
        finally:
            D.clusters_pay = real
        assert float((got[-1].double() - want).norm() / want.norm()) < 3e-3
