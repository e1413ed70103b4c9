"""The binding's nodes where no gradient arrives: as the Python functions."""
import pytest
import torch

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
