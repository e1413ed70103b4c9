"""The nodes that the binding records for sparse_dense_product and fixed_mask_attention: the gradients of the Python functions, bit by bit, and their ways with saved
tensors, with whatever listens, and with what they do not support."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from gpu_util import DEV, problem
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, VsError, cvse, ops, torch_ops

pytestmark = pytest.mark.gpu
SPARSE, ATTENTION = 0, 1


def half(*shape):
    return torch.randn(shape, device=DEV).half()


def setting(which, batch=0, shared=True, V=8):
    torch.manual_seed(3)
    lead = (batch,) if batch else ()
    if which == SPARSE:
        a = problem(cvse.GEN_BETA, 14, 256 // V, 192, V, 0.8)
        operands = [half(*(() if shared else lead), a.nnz_vec * V), half(*lead, 192, 128)]
        grad, extra = half(*lead, 256, 128), ()
    else:
        a = problem(cvse.GEN_BAND, 6, 512 // V, 512, V, 0.8, band=64)
        operands, grad, extra = [half(*lead, 512, 64) for _ in range(3)], half(*lead, 512, 64), (0.125,)
    return operands, (torch_ops.AttentionMask(a, DEV), *extra), grad


NATIVE = {SPARSE: torch_ops.sparse_dense_product, ATTENTION: torch_ops.fixed_mask_attention}
PYTHON = {SPARSE: torch_ops.SparseDenseProduct, ATTENTION: torch_ops.FixedMaskAttention}


def wanting(operands, wanted=None):
    return [t.detach().clone().requires_grad_(wanted is None or i in wanted) for i, t in enumerate(operands)]


@pytest.mark.parametrize("which,batch,shared", [(SPARSE, 0, True), (SPARSE, 3, True), (SPARSE, 3, False), (SPARSE, 1, True), (ATTENTION, 0, True), (ATTENTION, 2, True)])
@pytest.mark.parametrize("path", [VS_PATH_TENSOR, VS_PATH_CUDA_CORE])
def test_gradients_of_the_python_function(which, batch, shared, path):
    operands, rest, grad = setting(which, batch, shared)
    for wanted in [(0,), (1,), (0, 1), tuple(range(len(operands)))]:
        mine, theirs = wanting(operands, wanted), wanting(operands, wanted)
        a, b = NATIVE[which](*mine, *rest, path), PYTHON[which].apply(*theirs, *rest, path)
        assert a.grad_fn is not None and type(a.grad_fn) is not type(b.grad_fn)   # the node, not the function
        assert torch.equal(a, b)
        for g in (grad, grad.transpose(-1, -2).contiguous().transpose(-1, -2)):   # in another order too
            x = torch.autograd.grad(a, [mine[i] for i in wanted], g, retain_graph=True)
            y = torch.autograd.grad(b, [theirs[i] for i in wanted], g, retain_graph=True)
            assert all(torch.equal(p, q) for p, q in zip(x, y))
    with torch.no_grad():
        assert NATIVE[which](*wanting(operands), *rest, path).grad_fn is None


@pytest.mark.parametrize("which", [SPARSE, ATTENTION])
def test_saved_tensors(which):
    operands, rest, grad = setting(which)
    packed = []
    x = wanting(operands)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.to(DEV)):
        out = NATIVE[which](*x, *rest)
    assert len(packed) == len(operands)
    got = torch.autograd.grad(out, x, grad)
    y = wanting(operands)
    want = torch.autograd.grad(NATIVE[which](*y, *rest), y, grad)
    assert all(torch.equal(p, q) for p, q in zip(got, want))
    with pytest.raises(RuntimeError, match="second time|already been freed"):
        torch.autograd.grad(out, x, grad)
    z = [t.clone() for t in wanting(operands)]   # not leaves
    out = NATIVE[which](*z, *rest)
    z[1].mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(grad)


def test_listeners_and_derivatives_of_the_backward_pass(monkeypatch):
    operands, rest, grad = setting(SPARSE)

    class Listen(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func.namespace == "vsparse":
                self.seen.append(func.overloadpacket.__name__)
            return func(*args, **(kwargs or {}))
    x = wanting(operands)
    out = NATIVE[SPARSE](*x, *rest)
    with Listen():
        heard = torch.autograd.grad(out, x, grad, retain_graph=True)
    assert Listen.seen == ["sddmm"]
    want = torch.autograd.grad(out, x, grad, retain_graph=True)
    assert all(torch.equal(p, q) for p, q in zip(heard, want))
    assert all(torch.equal(p, q) for p, q in zip(torch.autograd.grad(out, x, grad, create_graph=True), want))

    def refuse(*args):
        raise VsError(-3, "vs_spmm_t")
    monkeypatch.setattr(ops, "spmm_t", refuse)
    with pytest.raises(VsError):   # of the same type through the node
        torch.autograd.grad(out, x, grad, create_graph=True)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as profile:
        with torch.no_grad():
            NATIVE[SPARSE](*x, *rest)
    assert any(e.key == "vsparse::spmm" for e in profile.key_averages())


@pytest.mark.parametrize("which", [SPARSE, ATTENTION])
def test_what_the_functions_do_not_support(which):
    operands, rest, _ = setting(which)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: NATIVE[which](t, *operands[1:], *rest))(torch.stack([operands[0]] * 2))
    import torch.autograd.forward_ad as fwd
    with pytest.raises((NotImplementedError, RuntimeError)), fwd.dual_level():
        NATIVE[which](fwd.make_dual(operands[0], operands[0]), *operands[1:], *rest)
    x = wanting([t.float() for t in operands])   # not fp16: refused as ever
    with pytest.raises((TypeError, VsError, ValueError)):
        NATIVE[which](x[0], *operands[1:], *rest)
