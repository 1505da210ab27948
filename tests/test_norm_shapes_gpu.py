"""Norm backward on both sides of the lines between its layouts (rows to a warp or to a block, with the next row's loads ahead
or not), with every type, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 8), (3, 768), (448, 512), (449, 512), (449, 768), (4096, 768), (4097, 768), (5000, 264), (700, 776), (600, 1024), (301, 1032), (1500, 2048), (900, 2056),
         (700, 4096), (300, 4104), (250, 6144)]


@pytest.mark.parametrize("rms", [False, True], ids=["layer", "rms"])
@pytest.mark.parametrize("dy_type,x_type", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
@pytest.mark.parametrize("rows,C", SIZES)
def test_norm_backward(rows, C, dy_type, x_type, rms):
    from infinitrain_b200 import _ext

    ext = _ext.load(required=True)
    torch.manual_seed(rows + C)
    x = torch.randn(rows, C, device="cuda").to(x_type)
    dy, dres = torch.randn(rows, C, device="cuda").to(dy_type), torch.randn(rows, C, device="cuda").to(x_type)
    gamma, beta = torch.randn(C, device="cuda"), torch.randn(C, device="cuda")
    xd, gd = x.double().requires_grad_(), gamma.double().requires_grad_()
    if rms:
        y = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * gd
    else:
        y = torch.nn.functional.layer_norm(xd, (C,), gd, beta.double(), 1e-5)
    want_dx, want_dg = torch.autograd.grad(y, (xd, gd), dy.double())
    for with_res in (False, True):
        slot = torch.ones(C, device="cuda") if with_res else None
        if rms:
            _, rstd = ext.rmsnorm_fwd(x, gamma, 1e-5, torch.float32)
            dx, dg, dsum = ext.rmsnorm_bwd(dy, x, gamma, rstd, dres if with_res else None, slot, None, with_res)
        else:
            _, mean, rstd = ext.layernorm_fwd(x, gamma, beta, 1e-5, torch.float32)
            dx, dg, db, dsum = ext.layernorm_bwd(dy, x, gamma, mean, rstd, True, dres if with_res else None, slot, None, None, with_res)
            assert (db.double() - dy.double().sum(0)).norm() <= 1e-5 * dy.double().sum(0).norm()
        exact = want_dx + dres.double() if with_res else want_dx
        # one rounding of the stored value, fp32 sums
        unit = 2.0 ** -8 if x_type == torch.bfloat16 else 2e-6
        assert (dx.double() - exact).norm() <= unit * exact.norm() + 1e-6 * dy.double().norm()
        assert (dg.double() - (1 if with_res else 0) - want_dg).norm() <= 1e-5 * want_dg.norm() + 1e-6 * C ** 0.5
        if with_res:
            assert (dsum.double() - dres.double().sum(0)).norm() <= 1e-5 * dres.double().sum(0).norm()
