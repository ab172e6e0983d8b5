"""Prompts of which more than values is wanted take the library call, which torch knows as an operator (no GPU)."""
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx
from torch.utils.flop_counter import FlopCounterMode

from apt_serve_b200._native import only_values


def seen(run):
    """What ``only_values`` says inside of a transform."""
    answers = []

    def f(x):
        answers.append(only_values(x))
        return x * 2
    run(f)
    assert answers
    return set(answers)


def test_plain_tensors():
    x = torch.ones(3, requires_grad=True)
    assert only_values(torch.ones(3), torch.nn.Parameter(torch.ones(3), requires_grad=False))
    assert not only_values(torch.ones(3), x)
    with torch.no_grad():
        assert only_values(torch.ones(3), x, torch.nn.Parameter(torch.ones(3)))
    with torch.inference_mode():
        assert only_values(torch.ones(3), x)
    with torch.device("cpu"):   # a mode that only places new tensors
        assert only_values(torch.ones(3))


def test_transforms_and_traces():
    x = torch.ones(3)
    with torch.no_grad():
        assert seen(lambda f: torch.func.vmap(f)(x)) == {False}
        assert seen(lambda f: torch.func.jvp(f, (x,), (x,))) == {False}
        assert seen(lambda f: torch.jit.trace(f, (x,), check_trace=False)) == {False}
        assert seen(lambda f: make_fx(f)(x)) == {False}
        assert not torch.compile(lambda t: t * 2 + (100 if only_values(t) else 0), backend="eager")(x).gt(50).any()
        with FakeTensorMode():
            assert not only_values(torch.ones(3))
        with FlopCounterMode(display=False):
            assert not only_values(x)
        with torch.autograd.forward_ad.dual_level():
            assert not only_values(torch.autograd.forward_ad.make_dual(x, x))
    assert seen(lambda f: torch.func.grad(lambda t: f(t).sum())(x)) == {False}
    assert only_values(x)
