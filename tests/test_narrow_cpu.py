"""What the few-row kernel (csrc/kernels/narrow_gemm.cu) takes and refuses, as far as the host decides it."""
import pytest
import torch

from rmlx_b200.ops import narrow
from rmlx_b200.ops.weights import LinearWeight, W_BF16


def _shifted(t: torch.Tensor, by: int) -> torch.Tensor:
    """The same values, contiguous, ``by`` elements after a 16-byte boundary."""
    room = torch.zeros(t.numel() + 16, dtype=t.dtype)
    start = (-room.data_ptr() % 16) // t.element_size() + by
    view = room[start:start + t.numel()].view(t.shape)
    return view.copy_(t)


def _spread(t: torch.Tensor) -> torch.Tensor:
    """The same values, rows apart."""
    room = torch.zeros(*t.shape[:-1], t.shape[-1] + 8, dtype=t.dtype)
    room[..., :t.shape[-1]] = t
    return room[..., :t.shape[-1]]


@pytest.mark.parametrize("kind", ["q4", "q8"])
@pytest.mark.parametrize("lead", [(), (3,)])
def test_tables_that_are_views(kind, lead):
    w = LinearWeight.from_dense(torch.randn(*lead, 32, 512), kind)
    assert narrow.supported(w)
    for name in ("w", "scales", "biases"):
        whole = getattr(w, name)
        for other in (_shifted(whole, 1), _spread(whole)):
            assert torch.equal(other, whole)
            assert not narrow.supported(LinearWeight(w.kind, **{**{n: getattr(w, n) for n in ("w", "scales", "biases")}, name: other}))
        again = _shifted(whole, 16 // whole.element_size())
        assert narrow.supported(LinearWeight(w.kind, **{**{n: getattr(w, n) for n in ("w", "scales", "biases")}, name: again}))
    assert not narrow.supported(LinearWeight(w.kind, w.w, w.scales.half(), w.biases.half()))


def test_bf16_weights():
    w = torch.randn(32, 128).to(torch.bfloat16)
    assert narrow.supported(LinearWeight(W_BF16, w))
    assert not narrow.supported(LinearWeight(W_BF16, _shifted(w, 1)))
    assert not narrow.supported(LinearWeight(W_BF16, _spread(w)))
    assert not narrow.supported(LinearWeight(W_BF16, w.float()))
    assert not narrow.supported(LinearWeight(W_BF16, w[:24])) and not narrow.supported(LinearWeight(W_BF16, w[:, :96].contiguous()))


def test_launcher_refuses_before_any_launch():
    """Addresses that 16-byte copies cannot read return -2, with no device to launch on."""
    from rmlx_b200 import _lib
    try:
        fn = _lib.cuda().rmlx_narrow_gemm
    except Exception as e:                         # noqa: BLE001
        pytest.skip(f"CUDA library not available: {e}")
    at = dict(w=1 << 20, scales=1 << 21, biases=1 << 22, x=1 << 23, norm=1 << 24)

    def call(kind, **over):
        p = {**at, **over}
        return fn(kind, p["w"], p["scales"], p["biases"], p["x"], 512, 1, None, None, 1, p["norm"], 1e-6, None, 0, 1 << 25, 32, 0,
                  4, 32, 512, 0, 0, 0, 0, None)

    for kind in (1, 2):
        for name in ("w", "scales", "biases", "x", "norm"):
            assert call(kind, **{name: at[name] + 8}) == -2, name
        assert call(kind, scales=None) == -2 and call(kind, biases=None) == -2


@pytest.mark.parametrize("form", ["expert_ffn", "pairs_ffn"])
def test_experts_narrower_than_the_scratch(monkeypatch, form):
    """A scratch sized for the widest layer of a model serves its narrower layers too: they take the columns that they fill. The
    kernels' places are taken by plain products, which hold the operands to the shapes that the kernels' wrappers ask for."""
    g = torch.Generator().manual_seed(3)
    rows, top, experts, d = 3, 2, 4, 64
    layers = [tuple(LinearWeight(W_BF16, 0.1 * torch.randn(experts, n, k, generator=g)) for n, k in ((2 * inner, d), (d, inner)))
              for inner in (96, 32)]

    def product(x, w, chosen, x_div, out, swiglu):
        assert x.shape[1] == w.k and out.shape[0] >= len(chosen) and out.shape[1] >= (w.n // 2 if swiglu else w.n)
        for i, e in enumerate(chosen):
            y = w.w[e] @ x[i // x_div].float()
            if swiglu:
                y = torch.nn.functional.silu(y[:w.n // 2]) * y[w.n // 2:]
            out[i, :y.numel()] = y
        return out

    monkeypatch.setattr(narrow, "group_pairs", lambda idx, *a, **kw: (idx, idx))
    monkeypatch.setattr(narrow, "narrow_gemm", lambda x, w, norm_w=None, eps=0., out=None, swiglu=False, offsets=None, order=None, x_div=1,
                        rows=None, pdl=False: product(x, w, idx.flatten().tolist(), x_div, out, swiglu))
    monkeypatch.setattr(narrow, "pairs_gemm", lambda x, w, idx, x_div, out, norm_w=None, eps=0., swiglu=False, pdl=False:
                        product(x, w, idx.flatten().tolist(), x_div, out, swiglu))
    monkeypatch.setattr(narrow, "combine", lambda y, idx, experts, wts, residual, out, pdl=False:
                        residual + (wts[..., None] * y[:, :d].unflatten(0, idx.shape)).sum(1))
    scratch = narrow.ExpertScratch(rows, top, *layers[0])
    for up, down in layers:
        x, idx = torch.randn(rows, d, generator=g), torch.randint(0, experts, (rows, top), generator=g)
        wts, res = torch.rand(rows, top, generator=g), torch.randn(rows, d, generator=g)
        got = getattr(narrow, form)(x, idx, wts, up, down, torch.ones(d), 1e-6, residual=res, out=None, scratch=scratch)
        want = res.clone()
        for r in range(rows):
            for s in range(top):
                gate, value = (up.w[idx[r, s]] @ x[r]).chunk(2)
                act = (torch.nn.functional.silu(gate) * value).to(torch.bfloat16).float()     # the buffer between the two is bf16
                want[r] += wts[r, s] * (down.w[idx[r, s]] @ act)
        assert torch.allclose(got, want, atol=1e-5)
