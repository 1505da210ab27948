"""The GEMM for outputs of at most one wave of 128 x 64 tiles: every order of the operands and every number of shares of the
contraction with every epilogue, at sizes with remainders, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): one row; ragged tiles and shares of unequal length; shares of one k-block; a row of clusters
SIZES = [(1, 8, 1544), (130, 72, 520), (257, 200, 1096), (96, 768, 512), (300, 1001, 640)]
KINDS = ["plain", "bias", "bias32", "residual", "residual32", "gelu", "dgelu", "unaligned", "unaligned32", "gelu_residual"]


@pytest.mark.parametrize("shares", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("b_mn", [False, True], ids=["b_k_major", "b_mn_major"])
@pytest.mark.parametrize("a_mn", [False, True], ids=["a_k_major", "a_mn_major"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("M,N,K", SIZES)
def test_small_gemm(M, N, K, kind, a_mn, b_mn, shares):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    torch.manual_seed(M + N + shares)
    ld = (N + 63) // 64 * 64 + (1 if "unaligned" in kind else 0)       # odd rows: element by element
    dtype = torch.float32 if "32" in kind else torch.bfloat16
    a = torch.randn(K, (M + 7) // 8 * 8, device="cuda").bfloat16()[:, :M]         # rows a multiple of 16 bytes apart
    b = torch.randn(K, (N + 7) // 8 * 8, device="cuda").bfloat16()[:, :N]
    bias = torch.randn(N, device="cuda")
    operand = torch.randn(M, ld, device="cuda").to(dtype)[:, :N]
    exact = a.double().t() @ b.double()
    flags = (C.GEMM_OUT_F32 if dtype == torch.float32 else 0) | (C.GEMM_MAY_SPLIT if shares else 0)
    if kind not in ("plain", "dgelu"):
        flags |= C.GEMM_BIAS
        exact = exact + bias.double()
    if "residual" in kind or "unaligned" in kind:
        flags |= C.GEMM_RESIDUAL
        exact = exact + operand.double()
    if "gelu" in kind:
        flags |= C.GEMM_DGELU if kind == "dgelu" else C.GEMM_GELU_DUAL
    outs = []
    for _ in range(2):
        out, out2 = (torch.full((M, ld), float("nan"), device="cuda", dtype=dtype) for _ in range(2))
        C.gemm(a if a_mn else a.t().contiguous(), a_mn, b if b_mn else b.t().contiguous(), b_mn, M, N, K, out,
               out2 if flags & C.GEMM_GELU_DUAL else None, bias, operand if flags & C.GEMM_RESIDUAL else None,
               operand if kind == "dgelu" else None, flags, shares)
        outs.append((out, out2))
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    out, out2 = outs[0]
    assert torch.equal(out[:, :N], outs[1][0][:, :N])          # the shares are added in one order
    assert torch.isnan(out[:, N:].float()).all()

    got = out[:, :N].double()
    unit = 1e-6 if dtype == torch.float32 else 2.0 ** -8      # the stored value's rounding; fp32 sums of K products
    if kind == "dgelu":
        h = operand.double().requires_grad_()
        (slope,) = torch.autograd.grad(torch.nn.functional.gelu(h, approximate="tanh").sum(), h)
        inner = 0.7978845608 * (1 + 3 * 0.044715 * h.detach() ** 2)     # of the tanh; its error is 2^-11
        more = 2.0 ** -11 * (0.5 + h.detach().abs() * inner) * exact.abs() + 1e-6 * K * slope.abs()
        assert ((got - exact * slope).abs() <= unit * (exact * slope).abs() + 1e-6 * K + more).all()
        return
    assert ((got - exact).abs() <= unit * exact.abs() + 1e-6 * K).all()
    if "gelu" in kind:
        act = torch.nn.functional.gelu(got, approximate="tanh")
        assert ((out2[:, :N].double() - act).abs() <= unit * act.abs() + 1e-6 * K + 2.0 ** -11 * got.abs()).all()
