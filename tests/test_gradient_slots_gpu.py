"""Gradients that kernels add to a flat buffer themselves: tied and untied embedding tables, fresh weight gradients."""
import pytest
import torch

from infinitrain_b200.autocast import AutocastGuard
from infinitrain_b200.datatype import DataType
from infinitrain_b200.device import DeviceType
from infinitrain_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _leaf(shape, slot):
    p = torch.nn.Parameter(torch.randn(shape, device="cuda") * 0.1)
    if slot:
        p.grad = p.main_grad = torch.zeros_like(p.detach())
    return p


def _tied_loss(table, pos, idx):
    with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
        x = F.embedding(idx, table, pos)
        return F.linear(torch.tanh(x), table).float().square().mean()


@pytest.mark.parametrize("how", ["plain", "hook", "post_hook", "ready_hook", "other_grad", "inputs"])
def test_tied_table(how):
    """The same gradient whoever adds it up, and hooks that see it whole."""
    torch.manual_seed(1)
    table, pos = _leaf((200, 64), True), _leaf((40, 64), True)
    table._itb_shared = True
    idx = torch.randint(0, 200, (3, 32), device="cuda")
    want_table, want_pos = torch.autograd.grad(_tied_loss(table, pos, idx), (table, pos))     # no slot is touched by this
    assert not table.main_grad.any() and not pos.main_grad.any() and want_table.any()
    seen = []
    if how == "hook":
        table.register_hook(lambda g: seen.append(g.clone()))
    elif how == "post_hook":
        table.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))
    elif how == "ready_hook":
        table._itb_grad_ready_hooks = [lambda p: None]
    elif how == "other_grad":
        table.grad = torch.zeros_like(table)
    loss = _tied_loss(table, pos, idx)
    loss.backward(inputs=[pos]) if how == "inputs" else loss.backward()
    # fp32 sums of the same bf16 products in another order
    close = lambda a, b: (a - b).norm() <= 1e-5 * b.norm()
    assert close(pos.grad, want_pos)
    assert not table.grad.any() if how == "inputs" else close(table.grad, want_table)
    if how in ("hook", "post_hook"):
        assert len(seen) == 1 and close(seen[0], want_table)


def test_untied_table_accumulates():
    table = _leaf((100, 64), True)
    idx = torch.randint(0, 100, (2, 16), device="cuda")
    for _ in range(2):
        F.embedding(idx, table).sum().backward()
    count = torch.zeros(100, device="cuda").index_add_(0, idx.flatten(), torch.ones(32, device="cuda"))
    assert torch.equal(table.grad, 2 * count[:, None].expand(100, 64))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("rows,N,K", [(0, 64, 128), (8, 72, 64), (200, 264, 72), (96, 9500, 1032), (4096, 256, 256), (300, 100, 64)])
def test_fresh_weight_gradient(rows, N, K, mode):
    """Stored or cleared and added to, whatever the split of the contraction: nothing of what was there before is left."""
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    old = C.get_gemm_mode()
    C.set_gemm_mode(mode)
    try:
        ld = (N + 7) // 8 * 8
        dy = torch.randn(rows, ld, device="cuda").bfloat16()[:, :N]
        x = torch.randn(rows, K, device="cuda").bfloat16()
        out = torch.full((N, K + 4), float("nan"), device="cuda")
        C.gemm(dy, True, x, True, N, K, rows, out[:, :K], None, None, None, None, C.GEMM_OUT_F32 | C.GEMM_ATOMIC | C.GEMM_FRESH, 0)
        exact = dy.double().t() @ x.double()
        assert ((out[:, :K] - exact).abs() <= 1e-6 * (exact.abs() + rows)).all() and torch.isnan(out[:, K:]).all()
    finally:
        C.set_gemm_mode(old)
    assert C.kernel_status() == 0


def _slot_with_hook(shape, name, log, later):
    """A parameter whose ready hook notes which of the slots in ``later`` still hold nothing at its place in the stream."""
    p = torch.nn.Parameter(torch.randn(shape, device="cuda") * 0.1)
    p.main_grad = torch.zeros_like(p.detach())
    later.append(p.main_grad)
    p._itb_grad_ready_hooks = [lambda q: log.append((name, p.main_grad.clone(), [s.clone() for s in later]))]
    return p


@pytest.mark.parametrize("op", ["linear", "linear_gelu", "mlp"])
def test_ready_hooks_run_between_the_launches(op):
    """A hook runs as soon as its own gradient has been launched, ahead of the kernels of the gradients that follow."""
    log, slots = [], []
    x = torch.randn(2, 40, 64, device="cuda").bfloat16().requires_grad_()
    make = lambda shape, name: _slot_with_hook(shape, name, log, slots)
    if op == "mlp":
        w_fc, b_fc, w_proj, b_proj = make((128, 64), "w_fc"), make((128,), "b_fc"), make((64, 128), "w_proj"), make((64,), "b_proj")
        order, places = ["w_proj", "b_proj", "w_fc", "b_fc"], [2, 3, 0, 1]
        run = lambda: F.mlp_gelu(x, w_fc, b_fc, w_proj, b_proj)
    else:
        w, b = make((72, 64), "w"), make((72,), "b")
        order, places = ["w", "b"], [0, 1]
        run = lambda: F.linear(x, w, b, gelu=op == "linear_gelu")
    with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
        y = run()
    y.backward(torch.randn_like(y))
    assert [name for name, _, _ in log] == order
    for k, (name, own, seen) in enumerate(log):
        assert torch.equal(own, slots[places[k]]) and own.any(), name          # written whole when the hook runs
        for later in places[k + 1:]:
            assert not seen[later].any(), (name, "ran after", order[places.index(later)])


def test_error_in_a_ready_hook_is_the_callers():
    w = torch.nn.Parameter(torch.randn(72, 64, device="cuda"))
    w.main_grad = torch.zeros_like(w.detach())

    def fail(p):
        raise KeyError("bucket")

    w._itb_grad_ready_hooks = [fail]
    x = torch.randn(40, 64, device="cuda").bfloat16()
    y = F.linear(x, w)
    with pytest.raises(KeyError, match="bucket"):
        y.backward(torch.randn_like(y))


def test_hook_of_the_accumulator_sees_the_gradient():
    """Hooks of the node that adds a table's gradient up (what a wrapper for data parallelism registers) get it whole."""
    table = _leaf((100, 64), True)
    node = table.expand_as(table).grad_fn.next_functions[0][0]
    seen = []
    node.register_prehook(lambda grads: seen.append(grads[0]))
    F.embedding(torch.randint(0, 100, (2, 16), device="cuda"), table).sum().backward()
    assert len(seen) == 1 and seen[0] is not None and torch.equal(seen[0], table.grad) and table.grad.any()


def test_embedding_gradient_off_the_16_byte_grid():
    """A gradient whose rows start anywhere is copied before the kernel reads it."""
    table = _leaf((100, 64), False)
    idx = torch.randint(0, 100, (2, 16), device="cuda")
    dout = torch.randn(2 * 16 * 64 + 1, device="cuda")[1:].view(2, 16, 64)
    assert dout.is_contiguous() and dout.data_ptr() % 16
    (got,) = torch.autograd.grad(F.embedding(idx, table), table, dout)
    want = torch.zeros(100, 64, device="cuda").index_add_(0, idx.flatten(), dout.view(-1, 64))
    assert (got - want).norm() <= 1e-6 * want.norm()
