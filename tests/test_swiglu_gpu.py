"""The SwiGLU that reads its two inputs where they are, against the one that reads a copy: the same kernel, so the same
bits, whatever the layout of the inputs and of the gradient."""
import pytest
import torch


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_for_kernel_are_laid_out_as_the_kernels_want_them(dtype):
    from infinitrain_b200.ops import functional as ops

    for width in (8, 12, 16, 20, 24):
        base = torch.randn(5, width).to(dtype)
        for rows in (base, base[:1], base[2:3]):
            for first in range(width - 7):
                x = rows[:, first:first + 8]
                y = ops._rows_for_kernel(x)
                assert torch.equal(x, y)
                assert y.stride(1) == 1 and y.stride(0) % 8 == 0 and y.data_ptr() % 16 == 0


def _layouts(rows, F, dtype):
    wide = torch.randn(rows, 2 * F + 24, device="cuda").to(dtype)
    yield torch.randn(rows, F, device="cuda").to(dtype), torch.randn(rows, F, device="cuda").to(dtype)
    yield wide[:, :F], wide[:, F:2 * F]                    # rows of one wider matrix
    narrow = torch.randn(rows, F + 4, device="cuda").to(dtype)
    yield narrow[:, :F], narrow[:, 4:]                     # rows a multiple of 4, not of 8 elements apart
    yield wide[:, 8:F + 8], torch.randn(rows, F, device="cuda").to(dtype)     # unequal row strides
    yield wide[:, 1:F + 1], wide[:, F + 3:2 * F + 3]       # off the 16-byte boundary
    yield torch.randn(F, rows, device="cuda").to(dtype).t(), wide[:, :F]      # columns contiguous
    yield wide[:1, :F].expand(rows, F), wide[:, :F]        # one row for all


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,F", [(1, 8), (7, 264), (300, 1032)])
def test_swiglu_pair_is_swiglu(rows, F, dtype):
    from infinitrain_b200.ops import functional as ops

    torch.manual_seed(rows)
    for a, b in _layouts(rows, F, dtype):
        for dout in (torch.randn(rows, F, device="cuda").to(dtype), torch.randn(F, rows, device="cuda").to(dtype).t(),
                     torch.randn(rows, F + 1, device="cuda").to(dtype)[:, 1:]):
            results = []
            for fn in (ops.swiglu_pair, ops.swiglu):
                x, y = a.detach().requires_grad_(), b.detach().requires_grad_()
                out = fn(x, y)
                results.append((out, *torch.autograd.grad(out, (x, y), dout)))
            assert all(torch.equal(p, q) for p, q in zip(*results))


class _AlignedOnly:
    """The extension's two entries with what their kernels want of a layout, on the CPU."""

    @staticmethod
    def _check(*tensors):
        for t in tensors:
            assert t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0

    def swiglu_fwd(self, a, b):
        self._check(a, b)
        return a * torch.nn.functional.silu(b)

    def swiglu_bwd(self, dout, a, b):
        self._check(dout, a, b)
        s = torch.sigmoid(b)
        return torch.cat([dout * b * s, dout * a * (s + b * s * (1 - s))], dim=1)


def test_swiglu_of_a_copy_hands_the_kernels_aligned_rows(monkeypatch):
    from infinitrain_b200.ops import functional as ops

    monkeypatch.setattr(ops, "_C", lambda: _AlignedOnly())
    F = 8
    for rows in (1, 3):
        wide = torch.randn(rows, 2 * F + 8)
        for ab in (wide[:, :2 * F], wide[:, 1:2 * F + 1], torch.randn(rows, 2 * F + 4)[:, 4:], torch.randn(2 * F, rows).t()):
            ab = ab.detach().requires_grad_()
            out = ops._SwiGLUFn.apply(ab)
            dout = torch.randn(rows, F + 8)[:, 3:F + 3]
            (got,) = torch.autograd.grad(out, ab, dout)
            a, b = ab.detach()[:, :F].requires_grad_(), ab.detach()[:, F:].requires_grad_()
            ref = a * torch.nn.functional.silu(b)
            assert torch.allclose(out, ref)
            assert torch.allclose(got, torch.cat(torch.autograd.grad(ref, (a, b), dout), dim=1), atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_swiglu_kernels_refuse_what_is_off_the_boundary(dtype):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    good, wide = torch.randn(4, 16, device="cuda").to(dtype), torch.randn(4, 24, device="cuda").to(dtype)
    off = wide[:, 1:17]         # the host looks at the pointer: nothing is launched
    with pytest.raises(RuntimeError):
        C.swiglu_fwd(off, off)
    with pytest.raises(RuntimeError):
        C.swiglu_bwd(off, good, good)
