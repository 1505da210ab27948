"""A row of a forward GEMM has the same bits whatever rows are computed beside it: every kernel walks the contraction in one
order, so that the sampler's logits do not depend on the batch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows on both sides of the lines between the kernels: 128 x 64 tiles, 128 x 256 tiles, CTA pairs
@pytest.mark.parametrize("kind", ["plain", "residual", "residual32", "gelu"])
@pytest.mark.parametrize("N,K", [(768, 768), (768, 3072), (3072, 768), (520, 1096), (1001, 640), (9480, 264)])
def test_rows_do_not_depend_on_their_number(N, K, kind):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    torch.manual_seed(N + K)
    most, ld = 2331, (N + 63) // 64 * 64
    dtype = torch.float32 if kind == "residual32" else torch.bfloat16
    a = torch.randn(most, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda")
    residual = torch.randn(most, ld, device="cuda").to(dtype)[:, :N]
    flags = {"plain": 0, "residual": C.GEMM_RESIDUAL, "residual32": C.GEMM_RESIDUAL | C.GEMM_OUT_F32, "gelu": C.GEMM_GELU_DUAL}[kind]
    whole = None
    for rows in (most, 1, 96, 129, 256, 1000):
        out, out2 = (torch.empty(rows, ld, device="cuda", dtype=dtype) for _ in range(2))
        C.gemm(a[:rows], False, b, False, rows, N, K, out, out2 if kind == "gelu" else None, bias,
               residual[:rows] if "residual" in kind else None, None, flags | C.GEMM_BIAS, 0)
        got = torch.cat((out[:, :N], out2[:, :N])) if kind == "gelu" else out[:, :N]
        if whole is None:
            whole = got
        else:
            want = torch.cat((whole[:rows], whole[most:most + rows])) if kind == "gelu" else whole[:rows]
            assert torch.equal(got, want), rows
    assert C.kernel_status() == 0


def test_only_gradients_are_split():
    """Splitting is the caller's to allow, whatever number of shares is asked for; a linear's input gradient allows it."""
    from infinitrain_b200 import _ext
    from infinitrain_b200.ops import functional as F

    C = _ext.load(required=True)
    torch.manual_seed(5)
    x = torch.randn(96, 3072, device="cuda").bfloat16()
    w = torch.randn(768, 3072, device="cuda").bfloat16()

    def product(flags, shares):
        out = torch.empty(96, 768, device="cuda", dtype=torch.bfloat16)
        C.gemm(x, False, w, False, 96, 768, 3072, out, None, None, None, None, flags, shares)
        return out

    whole, split = product(0, 0), product(C.GEMM_MAY_SPLIT, 0)
    assert torch.equal(product(0, 8), whole) and torch.equal(product(C.GEMM_MAY_SPLIT, 1), whole)
    assert torch.equal(product(C.GEMM_MAY_SPLIT, 8), split) and not torch.equal(split, whole)
    assert torch.equal(F.linear(x, w), whole)
    z = torch.zeros(96, 768, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    F.linear(z, w.t().contiguous()).backward(x)         # the same product as an input gradient
    assert torch.equal(z.grad, split)
