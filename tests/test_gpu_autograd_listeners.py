"""The binding's nodes where no gradient arrives, and where function modes or a tracer listen to the backward pass: as the Python functions."""
import pytest
import torch
from torch.overrides import TorchFunctionMode

from test_gpu_autograd_nodes import ATTENTION, NATIVE, PYTHON, SPARSE, setting, wanting

pytestmark = pytest.mark.gpu


class NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        return None


@pytest.mark.parametrize("which,batch,shared", [(SPARSE, 0, True), (SPARSE, 3, True), (SPARSE, 3, False), (ATTENTION, 0, True), (ATTENTION, 2, True)])
def test_no_gradient_arrives(which, batch, shared):
    """torch.autograd.Function makes zeros of it, and with them gradients of zeros."""
    operands, rest, _ = setting(which, batch, shared)
    for function in (PYTHON[which].apply, NATIVE[which]):
        x = wanting(operands)
        got = torch.autograd.grad(NoGradient.apply(function(*x, *rest)).sum(), x)
        assert all(g is not None and g.shape == t.shape and not g.any() for g, t in zip(got, x))


def test_function_modes_hear_the_backward_pass():
    """torch.autograd.grad itself is a function that the mode takes off its stack to run; the engine's own entry is not."""
    class Listen(TorchFunctionMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))
    operands, rest, grad = setting(SPARSE)
    seen = []
    for function in (PYTHON[SPARSE].apply, NATIVE[SPARSE]):
        x = wanting(operands)
        out = function(*x, *rest)
        with Listen() as mode:
            torch.autograd.Variable._execution_engine.run_backward((out,), (grad,), False, False, tuple(x), allow_unreachable=True, accumulate_grad=False)
        seen.append([f for f in mode.seen if "vsparse" in f])
    assert len(seen[0]) == 1 and seen[1] == seen[0]


def test_traces_hold_what_the_python_function_puts_there():
    """On the calling thread; a tracer does not follow the backward pass to the device's."""
    operands, rest, grad = setting(SPARSE)
    kinds = []
    for function in (PYTHON[SPARSE].apply, NATIVE[SPARSE]):
        x = wanting(operands, (0,))
        out = function(*x, *rest)
        engine = torch.autograd.Variable._execution_engine
        with torch.autograd.set_multithreading_enabled(False):
            trace = torch.jit.trace(lambda g: engine.run_backward((out,), (g,), True, False, (x[0],), allow_unreachable=True, accumulate_grad=False)[0], grad,
                                    check_trace=False)
        kinds.append([n.kind() for n in trace.graph.nodes() if n.kind().startswith("vsparse")])
    assert kinds[0] == ["vsparse::sddmm"] and kinds[1] == kinds[0]
