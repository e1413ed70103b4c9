"""The two transposed products of attention's backward (dV = P^T dO, dK = dS^T Q) in one launch: bit for bit what each gives by itself,
with one tile in all, a ragged last tile, and more tiles than the SMs that a product gets."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, captured_kernels, custom, dev, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [2, 4, 8])
@pytest.mark.parametrize("heads,n,d", [(3, 264, 128), (1, 64, 64), (3, 520, 64), (2, 264, 64), (100, 264, 64)])
@pytest.mark.parametrize("cores", [False, True])
def test_each_as_by_itself(monkeypatch, V, heads, n, d, cores):
    monkeypatch.setenv("VSPARSE_B200_SPMM_T", "gather" if cores else "dense")
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "fused")
    a = custom([4 * (7 * i % (n // 16)) for i in range(n // V)], n, V, seed=n + V)
    q, k, v, go = (dev(cvse.fill_random((heads, n, d), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0)) for i in range(4))
    gq, gk, gv, want_k, want_v = (torch.full((heads, n, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(5))
    ws_p, ws_g = (torch.zeros(heads, a.nnz_vec * V, dtype=torch.float16, device=DEV) for _ in range(2))
    s, t = structure(a), [dev(x) for x in cvse.transpose(a)]
    launches = captured_kernels(lambda: ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *s, *t, q, k, v, go, gq, gk, gv,
                                                                    ws_p, ws_g, 0.125))
    assert launches.count("spmm_dense_kernel") == (0 if cores else 1), launches
    assert launches.count("spmm_t_kernel") == (2 if cores else 1), launches
    ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *s, *t, q, k, v, go, gq, gk, gv, ws_p, ws_g, 0.125)
    for values, rhs, out in ((ws_g, q, want_k), (ws_p, go, want_v)):
        ops.spmm_t(a.m_vec, V, d, n, *t, values, rhs, out, a.nnz_vec)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(gk, want_k) and torch.equal(gv, want_v)


def test_of_the_composed_steps(monkeypatch):
    """The operators one after the other give the same two products, and still do where dQ or dK is written over dO or P."""
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "steps")
    monkeypatch.setenv("VSPARSE_B200_SPMM_T", "dense")   # tiles, whatever the density
    V, heads, n, d = 4, 2, 264, 64
    a = custom([4 * (7 * i % (n // 16)) for i in range(n // V)], n, V, seed=n + V)
    q, k, v, go = (dev(cvse.fill_random((heads, n, d), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0)) for i in range(4))
    s, t = structure(a), [dev(x) for x in cvse.transpose(a)]

    def run(over):
        grad_out = go.clone()
        ws_p, ws_g = (torch.zeros(heads * max(a.nnz_vec * V, n * d), dtype=torch.float16, device=DEV) for _ in range(2))
        p, g = (w[:heads * a.nnz_vec * V].view(heads, -1) for w in (ws_p, ws_g))
        gq, gk, gv = (torch.full((heads, n, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(3))
        if over in ("q on grad_out", "k on grad_out"):
            gq, gk = (grad_out, gk) if over[0] == "q" else (gq, grad_out)
        if over in ("q on p", "k on p"):
            at = ws_p[:heads * n * d].view(heads, n, d)
            gq, gk = (at, gk) if over[0] == "q" else (gq, at)
        launches = captured_kernels(lambda: ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *s, *t, q, k, v, grad_out, gq,
                                                                        gk, gv, p, g, 0.125))
        assert ops.device_status() == 0
        return launches.count("dense_plan_kernelILb1E"), [x.clone() for x in (gq, gk, gv)]

    plans, want = run("")
    assert plans == 1
    for over in ("q on grad_out", "k on grad_out", "q on p", "k on p"):
        plans, got = run(over)
        assert plans == 2
        assert all(torch.equal(x, w) for x, w in zip(got, want)), over
