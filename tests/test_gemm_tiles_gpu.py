"""GEMMs on both sides of the line between 128 x 64 and 256-wide tiles, at sizes with remainders, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): few enough 128 x 64 tiles for all SMs at once, whatever the mode ...
NARROW = [(1, 8, 8), (96, 768, 3072), (128, 64, 64), (129, 72, 72), (256, 3072, 768), (300, 1001, 200), (1152, 1024, 136),
          (2368, 512, 64)]
# ... and more: 256 x 256 tiles by CTA pairs (mode 1) or 128 x 256 tiles (mode 0)
WIDE = [(1153, 1024, 136), (2048, 640, 72), (300, 3200, 200), (1153, 1001, 136), (2331, 520, 72), (129, 9473, 64)]
CASES = [(*size, 1) for size in NARROW] + [(*size, mode) for size in WIDE for mode in (1, 0)]


@pytest.fixture
def C():
    from infinitrain_b200 import _ext

    mod = _ext.load(required=True)
    mode = mod.get_gemm_mode()
    yield mod
    mod.set_gemm_mode(mode)


@pytest.mark.parametrize("b_mn", [False, True], ids=["b_k_major", "b_mn_major"])
@pytest.mark.parametrize("M,N,K,mode", CASES)
def test_gemm_against_64_bits(C, M, N, K, mode, b_mn):
    C.set_gemm_mode(mode)
    torch.manual_seed(M + N)
    ld = (N + 63) // 64 * 64
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    bt = torch.zeros(K, ld, device="cuda", dtype=torch.bfloat16)
    bt[:, :N] = b.t()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, ld, device="cuda").bfloat16()[:, :N]
    exact = a.double() @ b.double().t() + bias.double()
    bt = bt[:, :N]          # rows of any length whose stride is a multiple of 8

    def run(flags, residual=None, dtype=torch.bfloat16, second=False, aux=None):
        outs = [torch.full((M, ld), float("nan"), device="cuda", dtype=dtype) for _ in range(1 + second)]
        C.gemm(a, False, bt if b_mn else b, b_mn, M, N, K, outs[0], outs[1] if second else None, bias, residual, aux,
               flags | C.GEMM_BIAS, 0)
        return [o[:, :N].double() for o in outs]

    def close(x, ref, unit, more=0.0):    # the stored value's rounding, and fp32 sums of K products
        assert ((x - ref).abs() <= unit * ref.abs() + 1e-6 * K + more).all()

    close(run(0)[0], exact, 2.0 ** -8)
    close(run(C.GEMM_OUT_F32, dtype=torch.float32)[0], exact, 1e-6)
    close(run(C.GEMM_RESIDUAL, residual=res)[0], exact + res.double(), 2.0 ** -8)
    res32 = torch.randn(M, ld, device="cuda")[:, :N]
    close(run(C.GEMM_OUT_F32 | C.GEMM_RESIDUAL, residual=res32, dtype=torch.float32)[0], exact + res32.double(), 1e-6)
    h = res.double().requires_grad_()
    (slope,) = torch.autograd.grad(torch.nn.functional.gelu(h, approximate="tanh").sum(), h)
    inner = 0.7978845608 * (1 + 3 * 0.044715 * h.detach() ** 2)       # of the tanh; its error is 2^-11
    close(run(C.GEMM_DGELU, aux=res)[0], exact * slope, 2.0 ** -8,
          2.0 ** -11 * (0.5 + h.detach().abs() * inner) * exact.abs() + 1e-6 * K * slope.abs())
    pre, act = run(C.GEMM_GELU_DUAL, second=True)
    close(pre, exact, 2.0 ** -8)
    close(act, torch.nn.functional.gelu(pre, approximate="tanh"), 2.0 ** -8, 2.0 ** -11 * pre.abs())   # tanh to 11 bits
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
