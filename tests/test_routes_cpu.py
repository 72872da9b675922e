"""Which kernel a call goes to where several take it (host arithmetic): points on both sides of the lines, at sizes that were timed on both
kernels."""
import pytest
import torch

from rmlx_b200.ops import decode as D, narrow, quantized as Q
from rmlx_b200.ops.weights import W_BF16, W_Q4, W_Q8


class _Weight:
    """A weight's kind and sizes; every table contiguous and at a 16-byte address."""

    def __init__(self, kind, n, k, experts=0):
        self.kind, self.n, self.k, self.experts = kind, n, k, experts


@pytest.fixture
def aligned(monkeypatch):
    monkeypatch.setattr(narrow, "supported", lambda w: True)


@pytest.mark.parametrize("tiles,hd,max_len,q8,pays", [
    (1, 128, 8192, False, True), (148, 128, 8192, False, True), (296, 64, 8192, False, True),
    (297, 128, 8192, False, False), (384, 128, 8192, False, False), (384, 128, 512, False, False), (448, 128, 8192, False, False),
    (512, 128, 8192, False, True), (592, 128, 8192, False, True), (640, 128, 8192, False, False), (640, 128, 1024, False, True),
    (1184, 128, 8192, False, False), (384, 128, 8192, True, True), (2400, 128, 8192, True, True), (384, 64, 8192, False, False),
    (512, 64, 1024, True, False)])
def test_decode_attention_tiles(tiles, hd, max_len, q8, pays):
    assert D.clusters_pay(tiles, hd, max_len, q8) is pays


def test_sixteen_blocks_merge_few_heads(monkeypatch):
    """Tiles of more than eight heads take clusters of up to eight blocks once there are more than four of them."""
    class _Plans:
        rmlx_flash_decode_gtiles = staticmethod(lambda hq, hkv: -(-hq // hkv // 16))
        rmlx_flash_decode_cluster_plan = staticmethod(lambda batch, tiles, max_len, hd, q8: 16 << 16 | tiles)

    monkeypatch.setattr(D._lib, "cuda", _Plans)
    assert D.cluster_plan(1, 64, 4, 128, 8192, False) == 16 << 16 | 4
    assert D.cluster_plan(2, 64, 4, 128, 8192, False) == 8 << 16 | 8
    assert D.cluster_plan(2, 64, 4, 128, 8192, True) == 16 << 16 | 8
    assert D.cluster_plan(2, 32, 4, 128, 8192, False) == 16 << 16 | 8


@pytest.mark.parametrize("rows,experts,n,k,row", [
    (9, 128, 3072, 4096, True), (128, 128, 3072, 4096, True), (191, 128, 3072, 4096, True), (192, 128, 3072, 4096, False),
    (256, 128, 4096, 1536, False), (176, 32, 4096, 2048, True), (224, 64, 2048, 2048, False), (224, 64, 2176, 2048, True), (32, 16, 1024, 1024, True),
    (33, 16, 1024, 1024, False), (33, 8, 512, 512, False), (33, 16, 2048, 1024, False), (33, 32, 1024, 1024, False),
    (191, 8, 4096, 7168, True), (33, 32, 2048, 1024, True)])
def test_experts_in_4_bits(rows, experts, n, k, row):
    """``rows`` of x for each expert: on tiles of W's rows, or of x's."""
    assert Q.row_pays(rows * experts, n, k, experts) is row


@pytest.mark.parametrize("n,k,most", [
    (4096, 2048, 72), (3072, 4096, 96), (8192, 1024, 0), (8192, 2048, 24), (6144, 2560, 36), (9472, 3072, 48), (8192, 4096, 72), (6144, 5120, 96),
    (8192, 14336, 96), (9600, 1024, 96), (12288, 4096, 96), (14336, 1024, 32), (16384, 1536, 64), (16384, 2048, 96), (24576, 512, 0),
    (32768, 512, 0), (32768, 1024, 32), (28672, 3072, 64), (28672, 4096, 96), (151936, 4096, 96), (2048, 2048, 0)])
def test_rows_of_4_bit_weights(n, k, most):
    """Up to ``most`` rows on tiles of W's rows."""
    assert [m for m in range(1, 160) if Q.row_pays(m, n, k)] == list(range(1, most + 1))


@pytest.mark.parametrize("kind,n,k,rows", [
    (W_Q4, 28672, 4096, (16,)), (W_Q4, 4096, 512, (16, 32)), (W_Q4, 6144, 1024, (16, 24)), (W_Q4, 8192, 1024, (16,)), (W_Q4, 8192, 2048, (16, 24)),
    (W_Q4, 8192, 3072, (16, 24, 32)), (W_Q4, 12288, 512, (16, 24)), (W_Q4, 12288, 1024, (16, 24, 32)), (W_Q4, 16384, 2048, (16,)),
    (W_Q8, 2048, 1024, (16, 24, 32)), (W_Q8, 4096, 2560, (16, 32)), (W_Q8, 4096, 3072, (32, 64)), (W_Q8, 2048, 4096, (32, 64)),
    (W_Q8, 8192, 512, (32,)), (W_Q8, 8192, 1024, (33, 64)), (W_Q8, 28672, 4096, (64,))])
def test_rows_on_the_weight_streaming_kernel(aligned, kind, n, k, rows):
    """Rows of 16, 17, 24, 25, 32, 33 and 64 that go there: all up to the largest of ``rows``."""
    w = _Weight(kind, n, k)
    assert [m for m in (1, 16, 17, 24, 25, 32, 33, 64, 65) if narrow.pays(w, m)] == [m for m in (1, 16, 17, 24, 25, 32, 33, 64) if m <= max(rows)]


@pytest.mark.parametrize("kind,n,k,streams", [
    (W_Q4, 16384, 2048, True), (W_Q4, 16384, 1024, False), (W_Q4, 8192, 8192, True), (W_Q4, 3584, 20480, True), (W_Q4, 3840, 18432, False),
    (W_Q4, 4096, 16384, False), (W_Q4, 4096, 20480, False), (W_Q4, 4096, 24576, True), (W_Q4, 4608, 24576, False), (W_Q4, 4608, 28672, True),
    (W_Q4, 5120, 16384, True), (W_Q8, 4096, 16384, True), (W_Q4, 2048, 32768, True), (W_Q4, 2048, 36864, False), (W_Q8, 4096, 36864, False)])
def test_one_row(aligned, kind, n, k, streams):
    """One row of a large quantised weight: the even split, or a block per 32 rows of W."""
    x = torch.zeros(1, 8, dtype=torch.bfloat16)
    assert D._several(1, _Weight(kind, n, k), x) is streams
    assert D._several(2, _Weight(kind, n, k), x) is True


@pytest.mark.parametrize("kind,experts,n,k,most", [
    (W_Q4, 128, 3072, 4096, 12), (W_Q8, 128, 3072, 4096, 14), (W_Q8, 32, 4096, 2048, 14), (W_Q4, 64, 2048, 2048, 12), (W_Q4, 16, 1024, 1024, 8),
    (W_Q8, 16, 1024, 1024, 8), (W_Q8, 32, 2048, 1024, 8), (W_BF16, 128, 3072, 4096, 0)])
def test_pairs_of_experts_on_the_weight_streaming_kernel(aligned, kind, experts, n, k, most):
    up, down = _Weight(kind, n, k, experts), _Weight(kind, k, n // 2, experts)
    assert [p for p in range(1, 20) if narrow.pays_grouped(up, down, p * experts)] == list(range(1, most + 1))


@pytest.mark.parametrize("kind,experts,d,inner,top,rows", [
    (W_Q4, 128, 4096, 1536, 8, (2, 3, 4)), (W_Q4, 128, 2048, 1024, 8, ()), (W_Q4, 64, 2048, 1024, 8, ()), (W_Q4, 64, 2048, 1024, 6, (5,)),
    (W_Q4, 64, 2048, 1536, 6, (3, 4, 5)), (W_Q4, 16, 8192, 4096, 2, (1, 2, 3)), (W_Q4, 16, 8192, 4096, 1, (2, 3, 4, 5, 6, 7)),
    (W_Q8, 16, 8192, 4096, 2, (1, 2, 3)), (W_Q8, 64, 2048, 1024, 8, (2, 3, 4)), (W_Q8, 64, 5120, 1536, 6, (1, 2, 3, 4, 5))])
def test_pairs_one_by_one(aligned, kind, experts, d, inner, top, rows):
    """Rows of a decode step, up to eight, whose pairs are multiplied one by one."""
    up, down = _Weight(kind, 2 * inner, d, experts), _Weight(kind, d, inner, experts)
    up.scales = down.scales = torch.zeros(1, dtype=torch.bfloat16)
    assert tuple(r for r in range(1, 9) if narrow.pays_pairs(up, down, r, top)) == rows


@pytest.mark.parametrize("kind,n,k,most", [(W_Q4, 151936, 4096, 160), (W_Q4, 32000, 2048, 160), (W_Q4, 50304, 1024, 160), (W_Q4, 65536, 512, 64),
                                           (W_Q4, 8192, 2048, 64), (W_Q4, 2048, 1024, 64), (W_Q8, 151936, 4096, 0)])
def test_logits_of_several_rows(kind, n, k, most):
    from rmlx_b200.models.prefill import _logits_by_rows
    assert max([r for r in range(200) if _logits_by_rows(_Weight(kind, n, k), r)], default=0) == most
