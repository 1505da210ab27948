"""GEMMs on both sides of the line between 128 x 64 and 256-wide tiles, at sizes with remainders, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): the first group has few enough 128 x 64 tiles for all SMs at once, the second has not
SIZES = [(1, 8, 8), (96, 768, 3072), (128, 64, 64), (129, 72, 72), (256, 3072, 768), (300, 1001, 200), (1152, 1024, 136),
         (2368, 512, 64), (1153, 1024, 136), (2048, 640, 72), (300, 3200, 200)]


@pytest.mark.parametrize("b_mn", [False, True], ids=["b_k_major", "b_mn_major"])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_gemm_against_64_bits(M, N, K, b_mn):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
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

    def run(flags, residual=None, dtype=torch.bfloat16, second=False):
        outs = [torch.full((M, ld), float("nan"), device="cuda", dtype=dtype) for _ in range(1 + second)]
        C.gemm(a, False, bt if b_mn else b, b_mn, M, N, K, outs[0], outs[1] if second else None, bias, residual, None,
               flags | C.GEMM_BIAS, 0)
        return [o[:, :N].double() for o in outs]

    def close(x, ref, unit, more=0.0):    # the stored value's rounding, and fp32 sums of K products
        assert ((x - ref).abs() <= unit * ref.abs() + 1e-6 * K + more).all()

    close(run(0)[0], exact, 2.0 ** -8)
    close(run(C.GEMM_OUT_F32, dtype=torch.float32)[0], exact, 1e-6)
    close(run(C.GEMM_RESIDUAL, residual=res)[0], exact + res.double(), 2.0 ** -8)
    pre, act = run(C.GEMM_GELU_DUAL, second=True)
    close(pre, exact, 2.0 ** -8)
    close(act, torch.nn.functional.gelu(pre, approximate="tanh"), 2.0 ** -8, 2.0 ** -11 * pre.abs())   # tanh to 11 bits
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
