"""Fixed-mask attention in one kernel per direction, at row lengths around its chunks of 32 keys, with each number of warps per
vector-row, against the fp64 oracle (conftest.assert_close), and the calls that it leaves to the operators."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, custom, dev, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu

# no keys, parts of a unit of 16, of a chunk of 32, of the chunks of two and four warps, and more than one round of those
LENS = [0, 1, 15, 16, 17, 31, 32, 33, 0, 63, 64, 65, 127, 128, 129, 200, 7]


def problem(V, d, heads):
    a = custom(LENS, 224, V, seed=V)
    rng = np.random.default_rng(V + d)
    a.col_indices[a.row_offsets[6]:a.row_offsets[7]] = rng.permutation(a.col_indices[a.row_offsets[6]:a.row_offsets[7]])   # unsorted
    q, go = (rng.standard_normal((heads, a.m, d)).astype(np.float16) for _ in range(2))
    k, v = (rng.standard_normal((heads, a.n, d)).astype(np.float16) for _ in range(2))
    return a, q, k, v, go


@pytest.mark.parametrize("warps", ["1", "2", "4"])
@pytest.mark.parametrize("V", [2, 4, 8])
@pytest.mark.parametrize("d", [64, 128])
def test_forward_and_backward(monkeypatch, V, d, warps):
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "fused")
    monkeypatch.setenv("VSPARSE_B200_ATTENTION_WARPS", warps)
    heads = 2
    a, q, k, v, go = problem(V, d, heads)
    scale = d ** -0.5
    st = structure(a)
    size = a.nnz_vec * V
    out, gq = (torch.full((heads, a.m, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(2))
    gk, gv = (torch.full((heads, a.n, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(2))
    ws_p, ws_g = (torch.full((heads * size + 64,), float("nan"), dtype=torch.float16, device=DEV) for _ in range(2))
    dq, dk, dv, dgo = (dev(x) for x in (q, k, v, go))
    ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, a.n, d, a.nnz_vec, *st, dq, dk, dv, out, ws_p, scale)
    probs = ws_p.float().cpu().numpy()
    t = [dev(x) for x in cvse.transpose(a)]
    ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, a.n, d, a.nnz_vec, *st, *t, dq, dk, dv, dgo, gq, gk, gv, ws_p, ws_g, scale)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert np.isnan(probs[heads * size:]).all() and bool(torch.isnan(ws_g[heads * size:]).all()), "wrote past the end"
    for h in range(heads):
        Q, K, Vm, G = (x[h].astype(np.float32) for x in (q, k, v, go))
        assert_close(out[h].float().cpu().numpy(), oracle.attention(a.m_vec, V, d, d, a.row_offsets, a.col_indices, Q, K, Vm, scale), "out")
        s = oracle.sddmm(a.m_vec, d, V, a.row_offsets, a.col_indices, Q, K, acc="f64")
        assert_close(probs[h * size:(h + 1) * size], oracle.softmax(a.m_vec, V, a.row_offsets, s, scale), "probabilities")
        want = oracle.attention_backward(a.m_vec, V, d, a.row_offsets, a.col_indices, Q, K, Vm, G, scale)
        for got, w, what in zip((gq, gk, gv), want, ("dQ", "dK", "dV")):
            assert_close(got[h].float().cpu().numpy(), w, what)


def test_a_non_finite_row_reaches_those_that_name_it(monkeypatch):
    """An Inf in a row of V and one in a row of K that few vector-rows name: the others keep their bits, also those whose last chunk is
    padded with a row they do not name (row 0 holds an Inf too)."""
    V, d = 8, 64
    a, q, k, v, _ = problem(V, d, 1)
    st = structure(a)
    ws = torch.empty(a.nnz_vec * V, dtype=torch.float16, device=DEV)

    def run(k, v):
        out = torch.empty((a.m, d), dtype=torch.float16, device=DEV)
        ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, a.n, d, a.nnz_vec, *st, dev(q[0]), dev(k), dev(v), out, ws, 0.125)
        torch.cuda.synchronize()
        return out.cpu().numpy().reshape(a.m_vec, V, d)

    clean = run(k[0], v[0])
    k1, v1 = k[0].copy(), v[0].copy()
    v1[0, 3] = np.inf
    k1[7, 5] = np.inf
    got = run(k1, v1)
    for i in range(a.m_vec):
        cols = a.col_indices[a.row_offsets[i]:a.row_offsets[i + 1]]
        if 0 in cols or 7 in cols:
            assert not np.isfinite(got[i].astype(np.float32)).all()
        else:
            assert np.array_equal(got[i], clean[i])


def test_operands_that_are_16_byte_aligned_only(monkeypatch):
    """The one-kernel form reads 32 bytes at a time; such operands go through the operators, with the same results to their rounding."""
    V, d = 8, 64
    a, q, k, v, _ = problem(V, d, 1)
    st = structure(a)
    want = oracle.attention(a.m_vec, V, d, d, a.row_offsets, a.col_indices, *(x[0].astype(np.float32) for x in (q, k, v)), 0.125)
    moved = []
    for x in (q, k, v):
        buf = torch.empty(x[0].size + 8, dtype=torch.float16, device=DEV)
        buf[8:] = dev(x[0]).view(-1)
        moved.append(buf[8:].view(x[0].shape))
    out = torch.empty((a.m, d), dtype=torch.float16, device=DEV)
    ws = torch.empty(a.nnz_vec * V, dtype=torch.float16, device=DEV)
    ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, a.n, d, a.nnz_vec, *st, *moved, out, ws, 0.125)
    torch.cuda.synchronize()
    assert_close(out.float().cpu().numpy(), want, "16-byte aligned")
