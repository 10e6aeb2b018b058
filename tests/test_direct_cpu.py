"""Which eager calls of the modules may skip the dispatcher (emmy_b200.linear._direct), decided on the CPU: the rule looks at the
thread's and the tensor's dispatch keys, so a plain CPU tensor's key set stands in for the CUDA one."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from emmy_b200 import linear


@pytest.fixture()
def x(monkeypatch):
    t = torch.zeros(2, 4)
    with torch.inference_mode():
        inference = torch.zeros(1)
    keys = {torch._C._dispatch_keys(t).raw_repr(), torch._C._dispatch_keys(inference).raw_repr()}
    monkeypatch.setattr(linear, "_PLAIN_KEYS", keys)
    return t


def test_plain_calls_are_direct(x):
    assert linear._direct(x)
    with torch.no_grad():
        assert linear._direct(x.clone().requires_grad_())
    with torch.inference_mode():
        assert linear._direct(torch.zeros(2, 4))


def test_calls_that_need_the_operator(x):
    seen = []

    def look(t):
        seen.append(linear._direct(t))
        return t * 1

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    look(x.clone().requires_grad_())  # gradients are recorded
    torch.func.vmap(look)(x)
    torch.func.jvp(look, (x,), (x,))
    torch.func.functionalize(look)(x)
    with torch.no_grad():
        torch.fx.experimental.proxy_tensor.make_fx(look)(x)
        torch.jit.trace(look, (x,), check_trace=False)
        with Mode():
            look(x)
        look(x.as_subclass(Sub))
        look(torch._neg_view(x))
        with torch._subclasses.FakeTensorMode():
            look(torch.zeros(2, 4))
        with torch.autograd.forward_ad.dual_level():
            look(torch.autograd.forward_ad.make_dual(x, x))
        with torch.device("cpu"):  # a function mode
            look(x)
        with torch.autograd.profiler.profile():
            look(x)
        assert not linear._direct(x, x)  # a weight that is not on a CUDA device
    assert len(seen) >= 12 and not any(seen)
