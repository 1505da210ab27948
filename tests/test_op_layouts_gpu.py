"""Linear, GELU MLP, norms and packed attention on the layouts that their entry points take: strided and expanded
tensors, rows off the 16-byte grid, odd widths, no rows, types that are converted; forward and gradients against the
reference formulation in fp32."""
import pytest
import torch

from infinitrain_b200.autocast import AutocastGuard
from infinitrain_b200.datatype import DataType
from infinitrain_b200.device import DeviceType
from infinitrain_b200.ops import functional as F
from infinitrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _layouts(shape, dtype):
    """The same values contiguous, with a wider row pitch, with transposed leading dimensions and off the 16-byte grid."""
    torch.manual_seed(sum(shape))
    base = torch.randn(shape, device="cuda").bfloat16().to(dtype)
    wide = torch.zeros(*shape[:-1], shape[-1] + 8, device="cuda", dtype=dtype)
    wide[..., :shape[-1]] = base
    odd = torch.zeros(*shape[:-1], shape[-1] + 3, device="cuda", dtype=dtype)
    odd[..., 1:shape[-1] + 1] = base
    return {"plain": base, "wide": wide[..., :shape[-1]], "transposed": base.transpose(0, 1).contiguous().transpose(0, 1),
            "odd": odd[..., 1:shape[-1] + 1]}


def _close(a, b, what):
    # bf16 operands, activations and stored results (2^-8 each), as 2-norms
    assert a.shape == b.shape and (a.double() - b.double()).norm() <= 1.2e-2 * b.double().norm() + 1e-6, what


def _compare(fused, plain, inputs, dy_layouts, what):
    leaves = [t.detach().clone().requires_grad_() if t is not None else None for t in inputs]
    expect = plain(*[t.float() if t is not None else None for t in leaves])
    for name, dy in dy_layouts(expect).items():
        want = torch.autograd.grad(expect, [t for t in leaves if t is not None], dy.float(), retain_graph=True)
        mine = [t.detach().requires_grad_() if t is not None else None for t in inputs]
        with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
            out = fused(*mine)
        _close(out.float(), expect, (what, "forward"))
        got = torch.autograd.grad(out, [t for t in mine if t is not None], dy.to(out.dtype))
        for a, b in zip(got, want):
            _close(a, b, (what, name))
        with torch.no_grad(), AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
            again = fused(*mine)
        assert torch.equal(out, again), (what, "without gradients")


def _dys(expect):
    return {"plain": torch.randn_like(expect).bfloat16(), "expanded": torch.ones((), device="cuda").bfloat16().expand_as(expect),
            "transposed": torch.randn_like(expect).bfloat16().transpose(0, 1).contiguous().transpose(0, 1)}


@pytest.mark.parametrize("layout", ["plain", "wide", "transposed", "odd"])
@pytest.mark.parametrize("N,bias,residual,gelu,dtype", [
    (96, True, None, False, torch.bfloat16), (100, True, None, True, torch.float32), (4, False, None, False, torch.bfloat16),
    (128, True, torch.bfloat16, False, torch.bfloat16), (72, True, torch.float32, False, torch.float32)])
def test_linear_layouts(layout, N, bias, residual, gelu, dtype):
    x = _layouts((3, 50, 80), dtype)[layout]
    w = torch.randn(N, 80, device="cuda").bfloat16().float() * 0.1
    b = torch.randn(N, device="cuda") if bias else None
    r = _layouts((3, 50, N), residual)["transposed"] if residual else None
    _compare(lambda x, w, b, r: F.linear(x, w, b, r, gelu), lambda x, w, b, r: ref.linear(x, w, b, r, gelu), [x, w, b, r], _dys,
             (layout, N))


@pytest.mark.parametrize("layout", ["plain", "wide", "transposed", "odd"])
@pytest.mark.parametrize("residual", [None, torch.bfloat16, torch.float32])
def test_mlp_layouts(layout, residual):
    x = _layouts((3, 50, 80), torch.bfloat16)[layout]
    w1, w2 = (torch.randn(*s, device="cuda").bfloat16().float() * 0.1 for s in ((160, 80), (80, 160)))
    b1, b2 = torch.randn(160, device="cuda"), torch.randn(80, device="cuda")
    r = _layouts((3, 50, 80), residual)["wide"] if residual else None
    plain = lambda x, w1, b1, w2, b2, r: ref.linear(ref.linear(x, w1, b1, None, True), w2, b2, r, False)
    _compare(F.mlp_gelu, plain, [x, w1, b1, w2, b2, r], _dys, layout)


@pytest.mark.parametrize("layout", ["plain", "wide", "transposed", "odd"])
@pytest.mark.parametrize("rope", [False, True])
def test_attention_layouts(layout, rope):
    H, KV, D, T = 4, 2, 64, 50
    qkv = _layouts((3, T, (H + 2 * KV) * D), torch.bfloat16)[layout]
    freqs = ref.precompute_freqs_cis(D, T + 7, 10000.0, torch.device("cuda")) if rope else None
    if layout in ("wide", "odd", "transposed") and not rope:
        if layout == "odd":         # the kernels read heads where they are: a projection off the 16-byte grid is refused
            with pytest.raises(RuntimeError):
                F.attention_packed(qkv, H, KV, D, None, 0, True)
            return
        out = F.attention_packed(qkv, H, KV, D, None, 0, True)
        assert torch.equal(out, F.attention_packed(qkv.contiguous(), H, KV, D, None, 0, True))
        return
    leaf = qkv.float().contiguous().requires_grad_()
    q, k, v = leaf.view(3, T, -1, D).split((H, KV, KV), dim=2)
    if rope:
        q, k = ref.apply_rope(q, freqs, 5), ref.apply_rope(k, freqs, 5)
    expect = ref.attention(q, k, v, True).reshape(3, T, H * D)
    for name, dy in _dys(expect).items():
        (want,) = torch.autograd.grad(expect, leaf, dy.float(), retain_graph=True)
        mine = qkv.detach().requires_grad_()
        out = F.attention_packed(mine.clone() if qkv.is_contiguous() else mine, H, KV, D, freqs, 5 if rope else 0, True)
        _close(out.float(), expect, layout)
        (got,) = torch.autograd.grad(out, mine, dy)
        _close(got, want, (layout, name))


def test_no_rows():
    x = torch.zeros(0, 7, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.randn(32, 64, device="cuda", requires_grad=True)
    y = F.linear(x, w)
    assert y.shape == (0, 7, 32)
    dx, dw = torch.autograd.grad(y, (x, w), torch.zeros_like(y))
    assert dx.shape == x.shape and not dw.any()


def test_gradient_slots_are_added_to():
    """Weights and biases with a slot in a flat gradient buffer: the kernels add to it and nothing comes back."""
    x = torch.randn(2, 40, 64, device="cuda").bfloat16().requires_grad_()
    w, b = torch.nn.Parameter(torch.randn(72, 64, device="cuda")), torch.nn.Parameter(torch.randn(72, device="cuda"))
    dy = torch.randn(2, 40, 72, device="cuda").bfloat16()
    with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
        dw, db = torch.autograd.grad(F.linear(x, w, b), (w, b), dy)
        fired = []
        w.main_grad, b.main_grad = torch.ones_like(w.detach()), torch.ones_like(b.detach())
        w._itb_grad_ready_hooks = b._itb_grad_ready_hooks = [lambda p: fired.append(p)]
        F.linear(x, w, b).backward(dy)
    assert w.grad is None and b.grad is None and [p is q for p, q in zip(fired, (w, b))] == [True, True]
    _close(w.main_grad - 1, dw, "weight")
    _close(b.main_grad - 1, db, "bias")


@pytest.mark.parametrize("T", [50, 800])           # 128 x 64 tiles, CTA pairs
@pytest.mark.parametrize("residual", [None, torch.bfloat16, torch.float32])
def test_one_row_for_all(T, residual):
    """Gradients, inputs and residuals that are one row expanded: the rows have no pitch that a tensor map could take."""
    torch.manual_seed(T)
    N, K = 640, 64
    row = lambda n, dtype: torch.randn(n, device="cuda").to(dtype).expand(3, T, n)
    w = torch.randn(N, K, device="cuda").bfloat16().float() * 0.1
    b = torch.randn(N, device="cuda")
    r = row(N, residual) if residual else None
    dys = lambda expect: {"one row": row(N, torch.bfloat16)}
    for x in (torch.randn(3, T, K, device="cuda").bfloat16(), row(K, torch.bfloat16)):
        _compare(lambda x, w, b, r: F.linear(x, w, b, r), lambda x, w, b, r: ref.linear(x, w, b, r, False), [x, w, b, r], dys, T)
    _compare(lambda x, w, b: F.linear(x, w, b, gelu=True), lambda x, w, b: ref.linear(x, w, b, None, True), [x, w, b], dys, T)


def test_sum_over_rows():
    """The gradient of a sum over all rows of a matrix."""
    x = torch.randn(300, 64, device="cuda").bfloat16().requires_grad_()
    w = torch.randn(72, 64, device="cuda", requires_grad=True)
    v = torch.randn(72, device="cuda").bfloat16()
    (F.linear(x, w).sum(0) * v).sum().backward()
    _close(x.grad, (v.float() @ w.detach().bfloat16().float()).expand(300, 64), "dx")
    _close(w.grad, v.float()[:, None] * x.detach().float().sum(0), "dw")
