"""The ops' forward is called directly only when autograd has nothing to record or to refuse."""
import pytest
import torch
from torch.autograd import forward_ad

from infinitrain_b200.ops import functional as ops


class _Twice(torch.autograd.Function):
    applied = 0

    @staticmethod
    def forward(ctx, x):
        _Twice.applied += not isinstance(ctx, ops._NoContext)
        ctx.save_for_backward(x)
        ctx.factor = 2
        return x * 2

    @staticmethod
    def backward(ctx, dy):
        return dy * 2


def _applied(fn):
    before = _Twice.applied
    fn()
    return _Twice.applied - before


def test_apply_is_left_out_only_without_gradients():
    x = torch.ones(3, requires_grad=True)
    assert _applied(lambda: ops._apply(_Twice, x)) == 1
    with torch.no_grad():
        assert _applied(lambda: ops._apply(_Twice, x)) == 0
        assert torch.equal(ops._apply(_Twice, x), x * 2)
        with forward_ad.dual_level():
            assert _applied(lambda: ops._apply(_Twice, x)) == 1
    with torch.inference_mode():
        assert _applied(lambda: ops._apply(_Twice, x)) == 0


def test_function_transforms_see_the_autograd_function():
    with torch.no_grad(), pytest.raises(RuntimeError):      # no setup_context: what apply refuses stays refused
        torch.vmap(lambda t: ops._apply(_Twice, t))(torch.ones(2, 3))


class _FilledElsewhere(torch.autograd.Function):
    """2 x + 1, written by something the tracer does not see, as a kernel launch is."""

    @staticmethod
    def forward(ctx, x):
        out = torch.empty_like(x)
        out.numpy()[...] = 2 * x.numpy() + 1
        return out

    @staticmethod
    def backward(ctx, dy):
        return 2 * dy


def test_a_trace_without_gradients_runs_the_function_again():
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: ops._apply(_FilledElsewhere, x), torch.ones(3), check_trace=False)
        assert torch.equal(traced(torch.full((3,), 5.0)), torch.full((3,), 11.0))


def test_a_profile_without_gradients_names_the_op():
    with torch.no_grad(), torch.autograd.profiler.profile() as prof:
        ops._apply(_Twice, torch.ones(3))
    assert "_Twice" in [event.name for event in prof.function_events]


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["gpt2", "llama3"])
def test_logits_are_the_same_with_and_without_gradients(family):
    from infinitrain_b200.autocast import AutocastGuard
    from infinitrain_b200.datatype import DataType
    from infinitrain_b200.device import DeviceType
    from infinitrain_b200.models import GPT2, LLaMA3
    from infinitrain_b200.parallel import global_env as genv
    from infinitrain_b200.parallel.process_group import ProcessGroupFactory

    if not genv.GlobalEnv.Instance().initialized:
        genv.InitAllEnv(world_size=1, rank=0)
        ProcessGroupFactory.Instance().Init()
    make, name = (GPT2, "gpt2") if family == "gpt2" else (LLaMA3, "llama3-1b")
    model = make(name, n_layer=1, vocab_size=1000, original_vocab_size=1000).to("cuda")
    x = torch.randint(0, 1000, (2, 77), device="cuda")
    with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
        with_gradients = model(x).detach()
        with torch.no_grad():
            assert torch.equal(model(x), with_gradients)
