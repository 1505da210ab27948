"""Fused ops behind ``torch.autograd.Function``: the CUDA path launches the hand-written sm_100a
kernels of ``infinitrain_b200._C``; the CPU path (and any dtype the kernels do not cover) runs the
PyTorch implementations of :mod:`infinitrain_b200.ops.reference`.

Mixed precision follows the reference's autocast policy at module granularity
(infini_train/include/autocast.h:36-71): Linear/Matmul run in bf16 with fp32 accumulation and emit
bf16, normalisation and softmax statistics are fp32, weight gradients are fp32.  The casts are not
materialised: weights have a bf16 shadow that the fused optimizer refreshes, and activations stay
bf16 between the fused kernels.
"""
from __future__ import annotations

import functools
from typing import Optional

import torch
from torch.autograd import forward_ad

from .. import _ext
from . import reference as ref

_counters = {"launches": 0}


def launch_count() -> int:
    """Number of native kernel launches issued through this module (for benchmarks)."""
    return _counters["launches"]


def _C():
    mod = _ext.load()
    if mod is None:
        raise RuntimeError("infinitrain_b200 native extension is not available")
    return mod


# --------------------------------------------------------------------------- autocast state
class _AutocastState:
    enabled = False
    dtype = torch.bfloat16


def autocast_enabled() -> bool:
    return _AutocastState.enabled


def autocast_dtype() -> torch.dtype:
    return _AutocastState.dtype


def _use_fused(x: torch.Tensor) -> bool:
    """Fused kernels run on CUDA when the activation is bf16 or bf16 autocast is on."""
    return x.is_cuda and (x.dtype == torch.bfloat16 or (_AutocastState.enabled and _AutocastState.dtype == torch.bfloat16))


# --------------------------------------------------------------------------- applying an op
class _NoContext:
    """Stands in for an autograd context when nothing is recorded."""

    def save_for_backward(self, *tensors):
        pass


def _apply(fn, *args):
    """``fn.apply(*args)``.  With gradients off and no function transform, forward-mode level or tracer active there
    is nothing for autograd to record or refuse, and the forward is called as it is: ``apply`` costs the host about
    5 us an op (12 layers of width 768 on 1 x 96 tokens, 87 ops, bound by the host: 2.71 -> 2.27 ms).
    A tracer records the applied function as a node that runs again; of a bare forward it would see the allocation of
    the output and nothing of the launch that fills it.  A profiler takes the op's name from ``apply``."""
    if (torch.is_grad_enabled() or torch._C._are_functorch_transforms_active() or forward_ad._current_level >= 0
            or torch._C._get_tracing_state() is not None or torch._C._autograd._profiler_enabled()):
        return fn.apply(*args)
    return fn.forward(_NoContext(), *args)


# --------------------------------------------------------------------------- bf16 weight shadows
def weight_lp(weight: torch.Tensor) -> torch.Tensor:
    """bf16 copy of an fp32 weight, cached on the tensor.

    The fused optimizers write the shadow in the same kernel as the fp32 update and stamp it with
    the weight's version; any other in-place change bumps the version and triggers a re-cast.
    """
    if weight.dtype == torch.bfloat16:
        return weight.detach()
    sh = getattr(weight, "_itb_shadow", None)
    ver = weight._version
    if sh is not None and getattr(weight, "_itb_shadow_version", -1) == ver and sh.device == weight.device:
        return sh
    if sh is None or sh.shape != weight.shape or sh.device != weight.device:
        sh = torch.empty_like(weight, dtype=torch.bfloat16)
    if weight.is_cuda and weight.is_contiguous():
        _C().cast_into(weight.detach(), sh)
        _counters["launches"] += 1
    else:
        sh.copy_(weight.detach())
    weight._itb_shadow = sh
    weight._itb_shadow_version = ver
    return sh


def mark_shadow_fresh(weight: torch.Tensor) -> None:
    """Called by fused optimizers after they wrote ``weight._itb_shadow`` themselves."""
    weight._itb_shadow_version = weight._version


def _pad_cols(n: int) -> int:
    return (n + 63) // 64 * 64


def _as_bf16_2d(x: torch.Tensor) -> torch.Tensor:
    """``x`` as a bf16 matrix whose rows the kernels can read."""
    return _C().bf16_rows(x)


# --------------------------------------------------------------------------- linear
class _LinearFn(torch.autograd.Function):
    """y = x W^T (+ bias) (+ residual), optionally y = gelu(x W^T + bias).

    Forward, dgrad and wgrad are three launches of the tcgen05 GEMM; bias / residual / GELU live in
    its epilogue, the weight gradient is accumulated in fp32 with split-K atomics, the bias
    gradient is a two-stage column sum.
    """

    @staticmethod
    def forward(ctx, x, weight, bias, residual, gelu):
        assert not gelu or residual is None, "gelu and residual epilogues are not combined"
        y, x2, pre = _C().linear_fwd(x, weight_lp(weight), bias, residual, gelu)
        _counters["launches"] += 1
        ctx.save_for_backward(x2, weight, pre)
        # the Parameter itself: its gradient may go straight to a flat buffer
        ctx.meta = (bias, claim_bias_grad(residual, bias), x.dtype, residual.dtype if residual is not None else None)
        return y

    @staticmethod
    def backward(ctx, dy):
        x2, weight, pre = ctx.saved_tensors
        bias, bias_elsewhere, x_dtype, res_dtype = ctx.meta
        need_x, need_w, need_b = ctx.needs_input_grad[:3]
        d_res = None
        if res_dtype is not None:
            d_res = dy if dy.dtype == res_dtype else dy.to(res_dtype)
        need_b = need_b and bias is not None and not bias_elsewhere
        main_w = _weight_slot(weight, ctx, 1) if need_w else None
        main_b = _main_grad_of(bias) if need_b else None
        # with GELU dy is the gradient of the activation: gelu'(h) is folded in with one pointwise pass
        dx, dw, db = _C().linear_bwd(dy, x2, weight_lp(weight) if need_x else None, pre, need_w, main_w, _ready(weight, main_w),
                                     need_b, main_b, _ready(bias, main_b))
        _counters["launches"] += (pre is not None) + need_x + need_w + 2 * need_b
        if dx is not None and x_dtype != torch.bfloat16:
            dx = dx.to(x_dtype)
        return dx, _for_autograd(weight, dw), db, d_res, None


def _weight_slot(weight, ctx=None, index=0):
    """The fp32 tensor that ``weight``'s gradient is added to by the kernel (flat DDP / ZeRO gradient buffers), or None."""
    if getattr(weight, "_itb_shared", False):
        # A parameter used by several ops (tied embedding / head): its ready hook must fire once, after the last
        # contribution, which is when autograd has visited all of them.
        return _accumulated_slot(ctx, index, weight) if ctx is not None else None
    main = getattr(weight, "main_grad", None)
    if main is None and getattr(weight, "_itb_main_grad_fn", None) is not None:
        main = weight._itb_main_grad_fn()
    return main


def _accumulated_slot(ctx, index, p):
    """The fp32 tensor that autograd would add the gradient of ``p`` to, the input of ``ctx``'s node whose edge is
    ``index``, when nobody looks at that gradient on its way there: a kernel may add to the tensor itself and hand nothing on.
    (The tied 50257 x 768 table of GPT-2: two gradients cleared, two additions, 0.26 ms a step.)  None with hooks (of the
    tensor or of its accumulator node), with another ``.grad`` than the slot or one off the 16-byte grid, in a pass that asks for the gradient itself (``torch.autograd.grad``) or leaves
    ``p`` out, and while the pass is recorded."""
    main = getattr(p, "main_grad", None)
    if (main is None or torch.is_grad_enabled() or getattr(p, "_itb_grad_ready_hooks", None)
            or getattr(p, "_itb_sp_hooked", False) or not _C().adds_in_place(p, main)):
        return None
    node = ctx.next_functions[index][0]
    try:
        return main if node is not None and torch._C._will_engine_execute_node(node) else None
    except RuntimeError:
        return None


def _ready(p, slot):
    """What a native pass calls once it has launched the kernel that adds ``p``'s gradient to ``slot``, or None."""
    if slot is None or not (getattr(p, "_itb_grad_ready_hooks", None) or getattr(p, "_itb_grad_elsewhere", False)):
        return None
    return functools.partial(_grad_written, p)


def _for_autograd(weight, dw):
    """``dw`` (None when the kernel has added it) in the type of ``weight``."""
    return dw if dw is None or weight.dtype == torch.float32 else dw.to(weight.dtype)


def _wgrad(C, dy2, x2, weight, N, K, M):
    """dW[N,K] = dy^T x in fp32.  Accumulates straight into ``weight.main_grad`` when the parameter
    has one (flat DDP / ZeRO gradient buffers) and then fires its grad-ready hooks."""
    main = _weight_slot(weight)
    dw = main if main is not None else torch.empty((N, K), device=dy2.device, dtype=torch.float32)
    flags = C.GEMM_OUT_F32 | C.GEMM_ATOMIC | (C.GEMM_FRESH if main is None else 0)
    C.gemm(dy2, True, x2, True, N, K, M, dw, None, None, None, None, flags, 0)
    _counters["launches"] += 1
    if main is None:
        return _for_autograd(weight, dw)
    _grad_written(weight)
    return None


def _main_grad_of(p: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """The fp32 slot of ``p`` in a flat gradient buffer that a kernel may accumulate into directly, or
    None (no flat buffer, or a parameter shared by several ops whose ready hook must fire once)."""
    if p is None or getattr(p, "_itb_shared", False):
        return None
    if getattr(p, "_itb_sp_hooked", False) or getattr(p, "_backward_hooks", None):
        return None      # a tensor hook must see this gradient (e.g. the sum over the tensor-parallel group)
    main = getattr(p, "main_grad", None)
    if main is None and getattr(p, "_itb_main_grad_fn", None) is not None:
        main = p._itb_main_grad_fn()
    if main is None or main.dtype != torch.float32 or not main.is_contiguous():
        return None
    return main


def autograd_ready_hook(fn):
    """Wraps a grad-ready callback for ``register_post_accumulate_grad_hook``: the call autograd makes
    for a parameter whose gradient another op will write later in this backward pass (see
    ``claim_bias_grad``) is dropped; that op reports the parameter through ``_itb_grad_ready_hooks``."""
    def hook(p):
        if getattr(p, "_itb_grad_elsewhere", False):
            return None
        return fn(p)
    return hook


def _grad_written(p: torch.Tensor) -> None:
    """A kernel has added ``p``'s gradient to its flat-buffer slot: tell the reducer / ZeRO group."""
    if getattr(p, "_itb_grad_elsewhere", False):
        p._itb_grad_elsewhere = False
    for hook in getattr(p, "_itb_grad_ready_hooks", ()):
        hook(p)


def _bias_grad(C, dy2, N):
    """Column sums of dY."""
    if N % 8 == 0 and dy2.data_ptr() % 16 == 0:
        _counters["launches"] += 2
        return C.colsum(dy2)
    return dy2.float().sum(0)


def linear(x, weight, bias=None, residual=None, gelu=False):
    """``x @ weight.T + bias`` with optional fused residual add or tanh-GELU."""
    K = x.shape[-1]
    if _use_fused(x) and K % 8 == 0 and weight.is_cuda:
        return _apply(_LinearFn, x, weight, bias, residual, gelu)
    if _AutocastState.enabled and x.dtype == torch.float32 and not x.is_cuda:
        # CPU emulation of the bf16 autocast of Linear: bf16-rounded operands, fp32 accumulate.
        y = ref.linear(x.to(_AutocastState.dtype).float(), weight.to(_AutocastState.dtype).float(), bias, None, gelu)
        return y if residual is None else y + residual
    return ref.linear(x, weight, bias, residual, gelu)


# --------------------------------------------------------------------------- fused GELU MLP
class _MlpGeluFn(torch.autograd.Function):
    """out = residual + gelu(x Wfc^T + bfc) Wproj^T + bproj as four GEMM launches forward+backward
    activations: the GELU is stored by the first GEMM's epilogue and its derivative is applied in the
    epilogue of the dgrad GEMM of the projection (reference composition:
    infini_train/src/nn/modules/transformer/mlp.cc:70-79)."""

    @staticmethod
    def forward(ctx, x, w_fc, b_fc, w_proj, b_proj, residual):
        y, x2, h, g = _C().mlp_gelu_fwd(x, weight_lp(w_fc), b_fc, weight_lp(w_proj), b_proj, residual)
        _counters["launches"] += 2
        ctx.save_for_backward(x2, h, g, w_fc, w_proj)
        ctx.meta = (b_fc, b_proj, claim_bias_grad(residual, b_proj), x.dtype, residual.dtype if residual is not None else None)
        return y

    @staticmethod
    def backward(ctx, dy):
        x2, h, g, w_fc, w_proj = ctx.saved_tensors
        b_fc, b_proj, bias_elsewhere, x_dtype, res_dtype = ctx.meta
        need_x, need_fc, need_bfc, need_proj, need_bproj = ctx.needs_input_grad[:5]
        d_res = None
        if res_dtype is not None:
            d_res = dy if dy.dtype == res_dtype else dy.to(res_dtype)
        need_bfc = need_bfc and b_fc is not None
        need_bproj = need_bproj and b_proj is not None and not bias_elsewhere
        main_fc = _weight_slot(w_fc) if need_fc else None
        main_proj = _weight_slot(w_proj) if need_proj else None
        main_bfc = _main_grad_of(b_fc) if need_bfc else None
        main_bproj = _main_grad_of(b_proj) if need_bproj else None
        dx, dw_fc, db_fc, dw_proj, db_proj = _C().mlp_gelu_bwd(
            dy, x2, h, g, weight_lp(w_fc), weight_lp(w_proj), need_x, need_fc, main_fc, _ready(w_fc, main_fc),
            need_bfc, main_bfc, _ready(b_fc, main_bfc), need_proj, main_proj, _ready(w_proj, main_proj),
            need_bproj, main_bproj, _ready(b_proj, main_bproj))
        _counters["launches"] += 1 + need_x + need_fc + need_proj + 2 * need_bfc + 2 * need_bproj
        if dx is not None and x_dtype != torch.bfloat16:
            dx = dx.to(x_dtype)
        return dx, _for_autograd(w_fc, dw_fc), db_fc, _for_autograd(w_proj, dw_proj), db_proj, d_res


def mlp_gelu(x, w_fc, b_fc, w_proj, b_proj, residual=None):
    if _use_fused(x) and x.shape[-1] % 8 == 0 and w_fc.shape[0] % 8 == 0:
        return _apply(_MlpGeluFn, x, w_fc, b_fc, w_proj, b_proj, residual)
    hmid = linear(x, w_fc, b_fc, gelu=True)
    return linear(hmid, w_proj, b_proj, residual=residual)


# --------------------------------------------------------------------------- normalisation
class _SkipHolder:
    """Travels on the skip tensor of a residual norm to the projection that adds it back in: that
    projection's bias gradient is the column sum of the skip's gradient, which the norm's backward
    kernel reads anyway."""

    __slots__ = ("bias",)

    def __init__(self):
        self.bias = None


def claim_bias_grad(residual, bias) -> bool:
    """Called by a linear whose epilogue adds ``residual``: True when the norm that produced
    ``residual`` as its skip output will compute ``bias``'s gradient (straight into the flat
    gradient buffer) in its own backward pass, so the linear must not."""
    holder = getattr(residual, "_itb_skip_holder", None)
    if holder is None or bias is None or holder.bias is not None or _main_grad_of(bias) is None:
        return False
    holder.bias = bias
    # Until that norm's backward has run, nothing may report this parameter's gradient as complete:
    # autograd still visits its accumulator (with an undefined gradient, because the linear returns
    # none) and fires the parameter's post-accumulate hook there, long before the norm writes the slot.
    bias._itb_grad_elsewhere = True
    return True


def _norm_param_grads(params, outs):
    """Gradient tensors for autograd, or None for parameters whose gradient the kernel has already
    added to their flat-buffer slot."""
    res = []
    for p, slot, g in zip(params, outs[0], outs[1]):
        if p is None:
            res.append(None)
        elif slot is not None:
            _grad_written(p)
            res.append(None)
        else:
            res.append(g)
    return res


class _LayerNormFn(torch.autograd.Function):
    """LayerNorm; with ``skip=True`` also returns the input as a second output, so that the residual
    connection around the normalised branch starts HERE: backward then receives the branch's
    gradient and the skip's gradient together and one kernel computes norm'(dy) + dskip (and the
    column sums of dskip for the bias of the projection that adds the skip back in)."""

    @staticmethod
    def forward(ctx, x, gamma, beta, eps, out_dtype, holder=None):
        C = _C()
        xc = x if x.is_contiguous() else x.contiguous()
        y, mean, rstd = C.layernorm_fwd(xc, gamma, beta, eps, out_dtype, type(ctx) is not _NoContext)
        _counters["launches"] += 1
        ctx.save_for_backward(xc, mean, rstd)
        ctx.params = (gamma, beta)
        ctx.holder = holder
        if holder is None:
            return y
        return y, xc.view_as(xc)

    @staticmethod
    def backward(ctx, dy, dskip=None):
        C = _C()
        x, mean, rstd = ctx.saved_tensors
        gamma, beta = ctx.params
        dyc = dy if dy.is_contiguous() else dy.contiguous()
        if dyc.dtype == torch.float32 and x.dtype == torch.bfloat16:
            dyc = dyc.to(torch.bfloat16)
        if dskip is not None:
            dskip = dskip if dskip.dtype == x.dtype else dskip.to(x.dtype)
            dskip = dskip if dskip.is_contiguous() else dskip.contiguous()
        bias = ctx.holder.bias if (ctx.holder is not None and dskip is not None) else None
        slots = (_main_grad_of(gamma), _main_grad_of(beta), _main_grad_of(bias))
        dx, dg, db, _ = C.layernorm_bwd(dyc, x, gamma, mean, rstd, beta is not None, dskip, slots[0],
                                        slots[1] if beta is not None else None, slots[2], False)
        _counters["launches"] += 2
        if bias is not None:
            _grad_written(bias)
        dgamma, dbeta = _norm_param_grads((gamma, beta), (slots, (dg, db)))
        return dx, dgamma, dbeta, None, None, None


class _RMSNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gamma, eps, out_dtype, holder=None):
        C = _C()
        xc = x if x.is_contiguous() else x.contiguous()
        y, rstd = C.rmsnorm_fwd(xc, gamma, eps, out_dtype, type(ctx) is not _NoContext)
        _counters["launches"] += 1
        ctx.save_for_backward(xc, rstd)
        ctx.params = (gamma,)
        ctx.holder = holder
        if holder is None:
            return y
        return y, xc.view_as(xc)

    @staticmethod
    def backward(ctx, dy, dskip=None):
        C = _C()
        x, rstd = ctx.saved_tensors
        (gamma,) = ctx.params
        dyc = dy if dy.is_contiguous() else dy.contiguous()
        if dyc.dtype == torch.float32 and x.dtype == torch.bfloat16:
            dyc = dyc.to(torch.bfloat16)
        if dskip is not None:
            dskip = dskip if dskip.dtype == x.dtype else dskip.to(x.dtype)
            dskip = dskip if dskip.is_contiguous() else dskip.contiguous()
        bias = ctx.holder.bias if (ctx.holder is not None and dskip is not None) else None
        slots = (_main_grad_of(gamma), _main_grad_of(bias))
        dx, dg, _ = C.rmsnorm_bwd(dyc, x, gamma, rstd, dskip, slots[0], slots[1], False)
        _counters["launches"] += 2
        if bias is not None:
            _grad_written(bias)
        (dgamma,) = _norm_param_grads((gamma,), ((slots[0],), (dg,)))
        return dx, dgamma, None, None, None


def _norm_out_dtype(x):
    if x.dtype == torch.bfloat16 or (_AutocastState.enabled and _AutocastState.dtype == torch.bfloat16):
        return torch.bfloat16
    return torch.float32


def _norm_fused(x, gamma) -> bool:
    C_ = x.shape[-1]
    return (x.is_cuda and x.dtype in (torch.float32, torch.bfloat16) and gamma.dtype == torch.float32 and C_ % 8 == 0
            and C_ <= 6144 and _ext.available())


def layernorm(x, gamma, beta=None, eps=1e-5):
    if _norm_fused(x, gamma):
        return _apply(_LayerNormFn, x, gamma, beta, eps, _norm_out_dtype(x))
    return ref.layernorm(x, gamma, beta, eps)


def rmsnorm(x, gamma, eps=1e-6):
    if _norm_fused(x, gamma):
        return _apply(_RMSNormFn, x, gamma, eps, _norm_out_dtype(x))
    return ref.rmsnorm(x, gamma, eps)


def layernorm_skip(x, gamma, beta=None, eps=1e-5):
    """``(layernorm(x), x)``: the second output is the start of the residual connection around the
    normalised branch.  Adding it back in through a fused linear's ``residual`` argument lets the
    backward pass add the skip's gradient inside the norm's backward kernel (no separate add) and
    take that linear's bias gradient from the same pass."""
    if _norm_fused(x, gamma):
        holder = _SkipHolder()
        y, xs = _apply(_LayerNormFn, x, gamma, beta, eps, _norm_out_dtype(x), holder)
        xs._itb_skip_holder = holder
        return y, xs
    return ref.layernorm(x, gamma, beta, eps), x


def rmsnorm_skip(x, gamma, eps=1e-6):
    """``(rmsnorm(x), x)``; see :func:`layernorm_skip`."""
    if _norm_fused(x, gamma):
        holder = _SkipHolder()
        y, xs = _apply(_RMSNormFn, x, gamma, eps, _norm_out_dtype(x), holder)
        xs._itb_skip_holder = holder
        return y, xs
    return ref.rmsnorm(x, gamma, eps), x


# --------------------------------------------------------------------------- activations
class _GeluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        xc = x if x.is_contiguous() else x.contiguous()
        ctx.save_for_backward(xc)
        _counters["launches"] += 1
        return _C().gelu_fwd(xc)

    @staticmethod
    def backward(ctx, dy):
        (x,) = ctx.saved_tensors
        dyc = dy.to(x.dtype)
        dyc = dyc if dyc.is_contiguous() else dyc.contiguous()
        _counters["launches"] += 1
        return _C().gelu_bwd(dyc, x)


def gelu(x):
    if x.is_cuda and x.dtype in (torch.float32, torch.bfloat16) and _ext.available():
        return _apply(_GeluFn, x)
    return ref.new_gelu(x)


def _rows_for_kernel(x: torch.Tensor) -> torch.Tensor:
    """``x`` as rows that the kernels can read in 16-byte pieces, a multiple of 8 elements apart (4 fp32 would be
    aligned too, but the kernels refuse it); a copy only when it is not laid out so."""
    x2 = x.reshape(-1, x.shape[-1])
    if x2.stride(-1) != 1 or x2.stride(0) % 8 or x2.data_ptr() % 16:
        x2 = x2.clone(memory_format=torch.contiguous_format)
    return x2


class _SwiGLUFn(torch.autograd.Function):
    """out = a * silu(b) for a, b the two column halves of one [rows, 2F] matrix."""

    @staticmethod
    def forward(ctx, ab):
        C = _C()
        F = ab.shape[-1] // 2
        ab2 = _rows_for_kernel(ab)
        out = C.swiglu_fwd(ab2[:, :F], ab2[:, F:])
        _counters["launches"] += 1
        ctx.save_for_backward(ab2)
        ctx.shape = ab.shape
        return out.view(*ab.shape[:-1], F)

    @staticmethod
    def backward(ctx, dout):
        C = _C()
        (ab2,) = ctx.saved_tensors
        F = ab2.shape[-1] // 2
        dab = C.swiglu_bwd(_rows_for_kernel(dout.to(ab2.dtype)), ab2[:, :F], ab2[:, F:])
        _counters["launches"] += 1
        return dab.view(ctx.shape)


def swiglu_packed(ab):
    """``ab[..., :F] * silu(ab[..., F:])`` for a packed [..., 2F] tensor."""
    F = ab.shape[-1] // 2
    if ab.is_cuda and ab.dtype in (torch.float32, torch.bfloat16) and F % 8 == 0 and _ext.available():
        return _apply(_SwiGLUFn, ab)
    return ref.swiglu(ab[..., :F], ab[..., F:])


class _SwiGLUPairFn(torch.autograd.Function):
    """out = a * silu(b) for two tensors of one shape and type, read where they are."""

    @staticmethod
    def forward(ctx, a, b):
        a2, b2 = _rows_for_kernel(a), _rows_for_kernel(b)
        if a2.stride(0) != b2.stride(0):       # the kernel has one row stride for both
            a2, b2 = (t if t.stride(0) == t.shape[1] else t.clone(memory_format=torch.contiguous_format)
                      for t in (a2, b2))
        out = _C().swiglu_fwd(a2, b2)
        _counters["launches"] += 1
        ctx.save_for_backward(a2, b2)
        ctx.shape = a.shape
        return out.view(a.shape)

    @staticmethod
    def backward(ctx, dout):
        a2, b2 = ctx.saved_tensors
        F = a2.shape[1]
        dab = _C().swiglu_bwd(_rows_for_kernel(dout.to(a2.dtype)), a2, b2)
        _counters["launches"] += 1
        return dab[:, :F].view(ctx.shape), dab[:, F:].view(ctx.shape)


def _swiglu_of_copy(a, b):
    if a.is_cuda and a.dtype in (torch.float32, torch.bfloat16) and a.shape[-1] % 8 == 0 and _ext.available():
        return _apply(_SwiGLUFn, torch.cat([a, b], dim=-1))
    return ref.swiglu(a, b)


def swiglu_pair(a, b):
    """``a * silu(b)`` for a caller that does not change ``a`` or ``b`` in place afterwards (both are kept for the
    backward pass; :func:`swiglu` keeps a copy).  2048 x 8192 in bf16: the copy takes as long as the kernel, 20 us."""
    if (a.is_cuda and a.dtype in (torch.float32, torch.bfloat16) and b.dtype == a.dtype and b.shape == a.shape
            and b.device == a.device and a.shape[-1] % 8 == 0 and a.numel() > 0 and _ext.available()):
        return _apply(_SwiGLUPairFn, a, b)
    return _swiglu_of_copy(a, b)


def swiglu(a, b):
    return _swiglu_of_copy(a, b)


# --------------------------------------------------------------------------- attention
class _AttentionFn(torch.autograd.Function):
    """Causal flash attention over a packed [B, T, (H + 2 KV) D] bf16 projection, with RoPE applied
    in place to the q and k heads first (and un-applied on their gradients)."""

    @staticmethod
    def forward(ctx, qkv, H, KV, D, freqs, pos0, causal):
        o, lse, qkv = _C().attention_packed_fwd(qkv, H, KV, D, freqs, pos0, causal)
        _counters["launches"] += 1 + (freqs is not None)
        ctx.save_for_backward(qkv, o, lse, freqs)
        ctx.meta = (H, KV, D, pos0, causal)
        return o

    @staticmethod
    def backward(ctx, dout):
        qkv, o, lse, freqs = ctx.saved_tensors
        H, KV, D, pos0, causal = ctx.meta
        dqkv = _C().attention_packed_bwd(dout, qkv, o, lse, H, KV, D, freqs, pos0, causal)
        _counters["launches"] += 4 + (freqs is not None)
        return dqkv, None, None, None, None, None, None


def attention_packed(qkv, n_head, n_kv_head, head_dim, freqs=None, pos0=0, causal=True):
    """Self-attention on a packed QKV projection ``[B, T, (H + 2 KV) D]`` -> ``[B, T, H D]``.

    ``freqs`` is the ``[T_max, D/2, 2]`` (cos, sin) table for rotary embedding or ``None``.
    On CUDA the packed buffer is rotated in place.
    """
    H, KV, D = n_head, n_kv_head, head_dim
    if qkv.is_cuda and D in (64, 128) and _use_fused(qkv):
        return _apply(_AttentionFn, qkv, H, KV, D, freqs, pos0, causal)
    B, T, _ = qkv.shape
    q = qkv[..., : H * D].reshape(B, T, H, D)
    k = qkv[..., H * D : (H + KV) * D].reshape(B, T, KV, D)
    v = qkv[..., (H + KV) * D :].reshape(B, T, KV, D)
    if freqs is not None:
        q = ref.apply_rope(q, freqs, pos0)
        k = ref.apply_rope(k, freqs, pos0)
    return ref.attention(q, k, v, causal).reshape(B, T, H * D)


# --------------------------------------------------------------------------- embedding
class _EmbeddingFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, idx, wte, wpe, pos0, vocab_start, out_dtype):
        C = _C()
        idx = idx if idx.is_contiguous() else idx.contiguous()
        out = C.embedding_fwd(idx, wte, wpe, pos0, vocab_start, out_dtype)
        _counters["launches"] += 1
        ctx.save_for_backward(idx, wte, wpe)
        ctx.meta = (pos0, vocab_start)
        return out

    @staticmethod
    def backward(ctx, dout):
        C = _C()
        idx, wte, wpe = ctx.saved_tensors
        pos0, vocab_start = ctx.meta
        dout = dout if dout.is_contiguous() else dout.contiguous()
        if dout.data_ptr() % 16:
            dout = dout.clone()
        # the kernel adds: to the tables' own gradients where it may, else to cleared ones that autograd adds on
        slots = [None, None]
        grads = [None, None]
        for i, table in enumerate((wte, wpe)):
            if table is not None and ctx.needs_input_grad[1 + i]:
                slots[i] = _accumulated_slot(ctx, 1 + i, table)
                if slots[i] is None:
                    slots[i] = grads[i] = torch.zeros_like(table, dtype=torch.float32, memory_format=torch.contiguous_format)
        C.embedding_bwd(idx, dout, *slots, pos0, vocab_start)
        _counters["launches"] += sum(s is not None for s in slots) + sum(g is not None for g in grads)
        return None, *grads, None, None, None


def embedding(idx, wte, wpe=None, pos0=0, vocab_start=0):
    """Token (+ position) embedding; ids outside ``[vocab_start, vocab_start + len(wte))`` give zero rows."""
    if wte.is_cuda and wte.dtype == torch.float32 and wte.shape[1] % 8 == 0 and idx.dim() == 2 and _ext.available():
        out_dtype = torch.bfloat16 if (_AutocastState.enabled and _AutocastState.dtype == torch.bfloat16) else torch.float32
        return _apply(_EmbeddingFn, idx, wte, wpe, pos0, vocab_start, out_dtype)
    return ref.embedding(idx, wte, wpe, pos0, vocab_start)


# --------------------------------------------------------------------------- cross entropy
class _CrossEntropyFn(torch.autograd.Function):
    """Mean softmax cross-entropy; the backward pass overwrites the logits buffer with dlogits."""

    @staticmethod
    def forward(ctx, logits, target):
        C = _C()
        V = logits.shape[-1]
        l2 = logits.reshape(-1, V) if logits.dim() != 2 else logits
        if l2.stride(-1) != 1:
            l2 = l2.contiguous()
        t = target.reshape(-1)
        t = t if t.is_contiguous() else t.contiguous()
        loss, lse, _ = C.ce_fwd(l2, t, V)
        _counters["launches"] += 1
        ctx.save_for_backward(l2, t, lse)
        ctx.shape = logits.shape
        return loss.reshape(())

    @staticmethod
    def backward(ctx, g):
        C = _C()
        l2, t, lse = ctx.saved_tensors
        V = l2.shape[-1]
        C.ce_bwd(l2, t, lse, g.reshape(1).float(), V, True)
        _counters["launches"] += 1
        return l2.view(ctx.shape), None


def cross_entropy(logits, target):
    """Mean cross-entropy over all rows.  On CUDA the logits tensor is consumed: after backward it
    holds the gradient."""
    if logits.is_cuda and logits.dtype in (torch.float32, torch.bfloat16) and _ext.available():
        return _CrossEntropyFn.apply(logits, target)
    return ref.cross_entropy(logits, target)
