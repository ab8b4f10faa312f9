"""ops.functional._call: the forward without autograd where nothing can be recorded, ``Function.apply`` everywhere else."""
import pytest
import torch
from torch.autograd import forward_ad

from tinyinfinitrain_b200.ops import functional as TF


class _Double(torch.autograd.Function):
    applied = 0

    @classmethod
    def apply(cls, *args):
        cls.applied += 1
        return super().apply(*args)

    @staticmethod
    def forward(ctx, x, w, fork):
        ctx.save_for_backward(x, w)
        ctx.set_materialize_grads(False)
        ctx.extra = fork
        y = x * w * 2
        return (y, x) if fork else y

    @staticmethod
    def backward(ctx, dy, dx=None):
        x, w = ctx.saved_tensors
        return dy * w * 2, (dy * x * 2).sum(), None


@pytest.fixture
def x():
    _Double.applied = 0
    return torch.arange(4.0, requires_grad=True)


W = torch.tensor(3.0)


def test_gradients_go_through_apply(x):
    y = TF._call(_Double, x, W, False)
    y.sum().backward()
    assert _Double.applied == 1 and torch.equal(x.grad, torch.full((4,), 6.0))


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_without_gradients_the_forward_runs_alone(x, mode):
    with mode():
        want, want_alias = _Double.apply(x, W, True)
        y, alias = TF._call(_Double, x, W, True)
        single = TF._call(_Double, x, W, False)
    assert _Double.applied == 1
    assert torch.equal(y, want) and torch.equal(single, want)
    for t, ref in ((y, want), (alias, want_alias), (single, want)):
        assert t.requires_grad == ref.requires_grad == False and t.grad_fn is None  # noqa: E712
    assert alias.data_ptr() == x.data_ptr() == want_alias.data_ptr()


def test_saved_tensor_hooks_see_nothing_either_way(x):
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t, lambda t: t), torch.no_grad():
        _Double.apply(x, W, False)
        TF._call(_Double, x, W, False)
    assert not packed


def test_forward_mode_is_still_refused(x):
    with torch.no_grad(), forward_ad.dual_level():
        dual = forward_ad.make_dual(x.detach(), torch.ones(4))
        with pytest.raises(RuntimeError):
            forward_ad.unpack_dual(TF._call(_Double, dual, W, False))
    assert _Double.applied == 1


def test_transforms_are_still_refused(x):
    with torch.no_grad(), pytest.raises(RuntimeError):
        torch.func.vmap(lambda v: TF._call(_Double, v, W, False))(x.detach())
    assert _Double.applied == 1


def test_a_tensor_that_left_its_transform_goes_through_apply(x):
    leaked = []
    torch.func.grad(lambda v: (leaked.append(v), v.sum())[1])(x.detach())
    with torch.no_grad():
        y = TF._call(_Double, leaked[0], W, False)
    assert _Double.applied == 1 and torch.equal(y, x.detach() * 6)


def test_a_trace_records_the_function(x):
    with torch.no_grad():
        try:
            torch.jit.trace(lambda v: TF._call(_Double, v, W, False), (x.detach(),), check_trace=False)
        except Exception:
            pass
    assert _Double.applied >= 1
