"""When an op may skip ``autograd.Function.apply``: only if nothing can need its backward or see the call."""
import torch

from archscale_b200.ops import backend


class _Square(torch.autograd.Function):
    applied = 0

    @staticmethod
    def forward(ctx, x):
        _Square.applied += not isinstance(ctx, backend.NoCtx)
        ctx.save_for_backward(x)
        return x * x

    @staticmethod
    def backward(ctx, g):
        (x,) = ctx.saved_tensors
        return 2 * x * g


def test_apply_skips_the_function_only_without_autograd_machinery():
    x = torch.randn(4, requires_grad=True)
    y = backend.apply(_Square, x)
    assert _Square.applied == 1 and torch.equal(torch.autograd.grad(y.sum(), x)[0], 2 * x)
    with torch.no_grad():
        z = backend.apply(_Square, x)
    assert _Square.applied == 1 and torch.equal(z, y) and not z.requires_grad
    with torch.inference_mode():
        assert backend.plain_call()


def test_transforms_and_traces_keep_the_function():
    seen = []

    def f(x):
        seen.append(backend.plain_call())
        return x + 1

    with torch.no_grad():
        torch.vmap(f)(torch.ones(2, 2))
        torch.jit.trace(f, torch.ones(2), check_trace=False)
        with torch.autograd.forward_ad.dual_level():
            f(torch.ones(2))
    assert seen == [False] * 3
    f(torch.ones(2))
    assert seen[-1] is False                                   # gradients on
