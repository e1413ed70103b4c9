"""Attention calls whose results lie on operands that the operators, one after the other, have read for the last time by then: same results as
with buffers of their own, whatever the call would take otherwise."""
import numpy as np
import pytest
import torch

from conftest import assert_close
import oracle
from gpu_util import DEV, dev, problem, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu
V, D, N, HEADS = 8, 64, 1024, 4


def operands():
    a = problem(cvse.GEN_BAND, 6, N // V, N, V, 0.8, band=64)
    return a, [dev(cvse.fill_random((HEADS, N, D), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0)) for i in range(4)]


def shifted(t, elems):
    """The tensor `elems` elements into a larger buffer, and a result that begins `elems` before it."""
    buf = torch.empty(t.numel() + elems, dtype=t.dtype, device=DEV)
    buf[elems:] = t.view(-1)
    return buf[elems:].view(t.shape), buf[:t.numel()].view(t.shape)


def test_output_over_the_keys():
    a, (q, k, v, _) = operands()
    want = [oracle.attention(a.m_vec, V, D, D, a.row_offsets, a.col_indices, *(x[h].float().cpu().numpy() for x in (q, k, v)), 0.125) for h in range(HEADS)]
    ws = torch.empty((HEADS, a.nnz_vec * V), dtype=torch.float16, device=DEV)
    for keys, out in ((k.clone(), None), shifted(k, 32 * D)):
        out = keys if out is None else out
        ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, N, D, a.nnz_vec, *structure(a), q, keys, v, out, ws, 0.125)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        for h in range(HEADS):
            assert_close(out[h].float().cpu().numpy(), want[h], f"head {h}")


@pytest.mark.parametrize("over", ["grad_out", "vmat"])
def test_gradient_of_the_queries_over_an_operand(over):
    a, (q, k, v, go) = operands()
    t = [dev(x) for x in cvse.transpose(a)]
    ws_p, ws_g = (torch.empty((HEADS, a.nnz_vec * V), dtype=torch.float16, device=DEV) for _ in range(2))
    got = {"grad_out": go, "vmat": v}[over].clone()
    gk, gv = (torch.empty_like(k) for _ in range(2))
    ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, N, D, a.nnz_vec, *structure(a), *t, q, k, got if over == "vmat" else v,
                                got if over == "grad_out" else go, got, gk, gv, ws_p, ws_g, 0.125)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for h in range(HEADS):
        want = oracle.attention_backward(a.m_vec, V, D, a.row_offsets, a.col_indices, *(x[h].float().cpu().numpy() for x in (q, k, v, go)), 0.125)
        for x, w, what in zip((got, gk, gv), want, ("dQ", "dK", "dV")):
            assert_close(x[h].float().cpu().numpy(), w, f"{what}, head {h}")
