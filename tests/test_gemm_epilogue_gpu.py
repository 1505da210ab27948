"""Epilogues of the CTA-pair GEMM when a pair has several tiles in turn (its staging slots, operand loads and accumulators
are used again), with ragged last tiles, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): more than 74 tiles of 256 x 256, with remainders of rows, of 64 and of 32 columns, and of column halves
SIZES = [(2100, 2320, 72), (4097, 1288, 64), (9473, 648, 40), (19000, 257, 64)]
KINDS = ["plain", "bias", "residual", "residual32", "residual32_bias", "gelu", "dgelu", "add", "gelu_residual", "unaligned32"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("M,N,K", SIZES)
def test_epilogue_over_several_tiles(M, N, K, kind):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    mode = C.get_gemm_mode()
    C.set_gemm_mode(1)
    torch.manual_seed(N + len(kind))
    ld = (N + 63) // 64 * 64
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda")
    exact = a.double() @ b.double().t()
    f32 = "32" in kind or kind == "add"
    dtype = torch.float32 if f32 else torch.bfloat16
    out = torch.full((M, ld), 2.0 if kind == "add" else float("nan"), device="cuda", dtype=dtype)
    out2 = torch.full((M, ld), float("nan"), device="cuda", dtype=dtype)
    # a row pitch that no tensor map takes: the epilogue's direct loads and stores
    operand = torch.randn(M, ld + 1 if kind == "unaligned32" else ld, device="cuda").to(dtype)[:, :N]
    flags = C.GEMM_OUT_F32 if f32 else 0
    if kind in ("bias", "residual32_bias", "gelu"):
        flags |= C.GEMM_BIAS
        exact = exact + bias.double()
    if "residual" in kind or kind == "unaligned32":
        flags |= C.GEMM_RESIDUAL
        exact = exact + operand.double()
    if kind == "add":
        flags |= C.GEMM_ATOMIC
        exact = exact + 2.0
    if "gelu" in kind:
        flags |= C.GEMM_DGELU if kind == "dgelu" else C.GEMM_GELU_DUAL
    try:
        for _ in range(1 if kind == "add" else 2):      # the second launch finds the slots' and barriers' last state gone
            C.gemm(a, False, b, False, M, N, K, out, out2 if kind.startswith("gelu") else None, bias,
                   operand if flags & C.GEMM_RESIDUAL else None, operand if kind == "dgelu" else None, flags, 0)
        torch.cuda.synchronize()
        assert C.kernel_status() == 0
    finally:
        C.set_gemm_mode(mode)

    got = out[:, :N].double()
    unit = 1e-6 if f32 else 2.0 ** -8           # the stored value's rounding; fp32 sums of K products
    if kind == "dgelu":
        h = operand.double().requires_grad_()
        (slope,) = torch.autograd.grad(torch.nn.functional.gelu(h, approximate="tanh").sum(), h)
        inner = 0.7978845608 * (1 + 3 * 0.044715 * h.detach() ** 2)     # of the tanh; its error is 2^-11
        more = 2.0 ** -11 * (0.5 + h.detach().abs() * inner) * exact.abs() + 1e-6 * K * slope.abs()
        assert ((got - exact * slope).abs() <= unit * (exact * slope).abs() + 1e-6 * K + more).all()
        return
    assert ((got - exact).abs() <= unit * exact.abs() + 1e-6 * K).all()
    if kind.startswith("gelu"):
        act = torch.nn.functional.gelu(got, approximate="tanh")
        assert ((out2[:, :N].double() - act).abs() <= unit * act.abs() + 1e-6 * K + 2.0 ** -11 * got.abs()).all()
    # bulk stores of bf16 end on 16 bytes; nothing is written beyond, and beyond N by fp32 with a residual or a sum
    end = N if f32 else (N + 7) // 8 * 8
    for o in (out, out2) if kind.startswith("gelu") else (out,):
        assert (o[:, end:] == 2.0).all() if kind == "add" else torch.isnan(o[:, end:].float()).all()


@pytest.mark.parametrize("M", [64, 40960])        # 128 x 64 tiles, CTA pairs
def test_gelu_derivative_far_from_zero(M):
    """1 and 0 as far as the square of the input is finite: the cube is not from 7e12 on."""
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    one = torch.zeros(M, 64, device="cuda", dtype=torch.bfloat16)
    one[:, 0] = 1
    far = torch.logspace(1, 19, 32, device="cuda")
    h = torch.cat((far, -far)).bfloat16().expand(M, 64).contiguous()
    out = torch.full((M, 64), float("nan"), device="cuda", dtype=torch.bfloat16)
    C.gemm(one, False, one[:64], False, M, 64, 64, out, None, None, None, h, C.GEMM_DGELU, 0)      # the product is 1
    assert torch.equal(out, (h > 0).bfloat16())
    assert C.kernel_status() == 0
