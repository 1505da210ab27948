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
