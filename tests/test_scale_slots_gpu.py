"""4-bit GEMMs whose blocks run several tiles: a slot of scales that is given back before its values have arrived is overwritten with those of a
later block of K. Every result repeats to the bit and lies within 3e-3 (bf16 rounding, 2^-9 at most each) of the 64-bit product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,bn,residual", [(1500, 2048, 4096, 64, True), (300, 8192, 4096, 64, True), (1500, 2048, 2048, 64, False),
                                               (1500, 4096, 2048, 128, True), (2000, 6144, 2048, 256, True), (2048, 8192, 2048, 0, True),
                                               (64, 40960, 1024, 0, True)])
def test_results_repeat(m, n, k, bn, residual):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from rmlx_b200.ops.gemm import GemmStatus
    from rmlx_b200.ops.quantized import xgemm
    from rmlx_b200.ops.weights import LinearWeight
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(m + n)
    w = LinearWeight.random(n, k, "q4", dev, generator=g)
    x = torch.randn(m, k, device=dev, generator=g).to(torch.bfloat16)
    r = torch.randn(m, n, device=dev, generator=g).to(torch.bfloat16) if residual else None
    want = x.double() @ w.dequantized().to(torch.bfloat16).double().t()
    if residual:
        want += r.double()
    first = xgemm(x, w, residual=r, bn=bn)
    assert float((first.double() - want).norm() / want.norm()) < 3e-3
    assert all(torch.equal(first, xgemm(x, w, residual=r, bn=bn)) for _ in range(40))
    GemmStatus.check(dev)
