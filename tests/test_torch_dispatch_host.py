"""The autograd functions reach their operators through torch's dispatcher wherever something listens there: a dispatch mode
(tracers are modes too), a profiler or a tensor subclass sees torch.ops.vsparse.* and can take the call.  The mode answers for the
kernels, so most of it needs no GPU."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from vectorsparse_b200 import cvse, torch_ops


class Answer(TorchDispatchMode):
    """Answers the library's operators with ones of the right shape and lists their names."""

    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func.namespace != "vsparse":
            return func(*args, **(kwargs or {}))
        self.seen.append(func.overloadpacket.__name__)
        if func is torch.ops.vsparse.attention.default:
            return torch.ones_like(args[7])
        _, m_vec, V = args[:3]
        if func is torch.ops.vsparse.spmm.default:
            return args[6].new_ones((m_vec * V, args[7].shape[-1]))
        return args[7].new_ones((args[3] * V,))


@pytest.fixture(params=["cpu", pytest.param("cuda:0", marks=pytest.mark.gpu)])
def mask(request):
    return torch_ops.AttentionMask(cvse.generate(cvse.GEN_UNIFORM, 1, 8, 64, 8, 0.5), request.param)


def zeros(mask, *shape):
    return torch.zeros(shape, dtype=torch.float16, device=mask.row_offsets.device)


def test_a_dispatch_mode_sees_the_operators(mask):
    q = zeros(mask, 1, 64, 64).requires_grad_(True)
    values = zeros(mask, mask.nnz_vec * 8).requires_grad_(True)
    with Answer() as mode:
        out = torch_ops.fixed_mask_attention(q, q, q, mask, 0.125)
        c = torch_ops.sparse_dense_product(values, zeros(mask, 64, 64), mask)
        g, = torch.autograd.grad(c, values, torch.ones_like(c))
    assert mode.seen == ["attention", "spmm", "sddmm"]
    assert bool((out == 1).all()) and c.shape == (64, 64) and g.shape == values.shape


def test_a_tensor_subclass_takes_the_call(mask):
    class Wrapped(torch.Tensor):
        seen = []

        @classmethod
        def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
            if func.namespace == "vsparse":
                cls.seen.append(func.overloadpacket.__name__)
                return zeros(mask, 64, 64)
            with torch._C._DisableTorchDispatch():
                return func(*args, **(kwargs or {}))

    torch_ops.sparse_dense_product(zeros(mask, mask.nnz_vec * 8).as_subclass(Wrapped), zeros(mask, 64, 64), mask)
    assert Wrapped.seen == ["spmm"]


@pytest.mark.gpu
@pytest.mark.parametrize("pre_dispatch", [False, True])
def test_a_trace_keeps_the_operator(pre_dispatch):
    """make_fx records the product, whichever of its two mode stacks the tracer sits on."""
    from torch.fx.experimental.proxy_tensor import make_fx
    mask = torch_ops.AttentionMask(cvse.generate(cvse.GEN_UNIFORM, 1, 8, 64, 8, 0.5), "cuda:0")
    values, b = torch.randn(mask.nnz_vec * 8, device="cuda:0").half(), torch.randn(64, 64, device="cuda:0").half()
    traced = make_fx(lambda v, x: torch_ops.sparse_dense_product(v, x, mask), pre_dispatch=pre_dispatch)(values, b)
    assert any(n.target is torch.ops.vsparse.spmm.default for n in traced.graph.nodes)
    assert torch.equal(traced(2 * values, b), torch_ops.sparse_dense_product(2 * values, b, mask))


def test_host_tensors_have_no_kernel():
    mask = torch_ops.AttentionMask(cvse.generate(cvse.GEN_UNIFORM, 1, 8, 64, 8, 0.5), "cpu")
    with pytest.raises(NotImplementedError):
        torch_ops.sparse_dense_product(zeros(mask, mask.nnz_vec * 8), zeros(mask, 64, 64), mask)
