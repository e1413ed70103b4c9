"""Sums that a multiplying kernel hands on to the kernel behind it: the answer is that kernel's, and what the multiplying kernel says
about it stands in a word of its own (the grid that reads "this call is mine" must not change it: its CTAs start and end at different
times).  The plan header is read from a caller's workspace: word 0 "mine", words 1 and 2 "redo" of the plan's first and second product."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, custom, dev, spmm_inputs, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu


def words(workspace):
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    return workspace[:12].cpu().numpy().view(np.int32).tolist()


# pairs of CTAs, single CTAs, and A laid out in memory in front of the pairs
@pytest.mark.parametrize("V,N,laid_out", [(8, 256, "plan"), (8, 64, "plan"), (2, 256, "plan"), (2, 256, "laid-out")])
def test_a_product(monkeypatch, V, N, laid_out):
    monkeypatch.setenv("VSPARSE_B200_SPMM_PAIR", "1")
    monkeypatch.setenv("VSPARSE_B200_SPMM_A", laid_out)
    a = custom([30] * (512 // V), 200, V, seed=3)
    unused = 199
    for i in range(a.m_vec):   # no vector-row names the last column
        row = a.col_indices[a.row_offsets[i]:a.row_offsets[i + 1]]
        if row[-1] == unused:
            row[-1] = next(c for c in range(198, -1, -1) if c not in row)
            row.sort()
    vals, B = spmm_inputs(a, N, np.float16, 11, sigma=0.5)
    workspace = torch.zeros(8 << 20, dtype=torch.uint8, device=DEV)

    def run(mode, rhs):
        monkeypatch.setenv("VSPARSE_B200_SPMM", mode)
        out = torch.full((a.m, N), float("nan"), dtype=torch.float16, device=DEV)
        ops.spmm.wmmaSpmm(a.m_vec, V, N, a.n, *structure(a), dev(vals), dev(rhs), out)
        torch.cuda.synchronize()
        return out

    bad = B.copy()
    bad[unused, 5] = np.inf
    ops.set_workspace(workspace)
    try:
        run("dense", B)
        assert words(workspace) == [1, 0, 0]
        got = run("dense", bad)
        assert words(workspace) == [1, 1, 0]
        run("dense", B)
        assert words(workspace) == [1, 0, 0]
    finally:
        ops.set_workspace(None)
    assert bool(torch.isfinite(got).all())
    assert torch.equal(got, run("gather", bad))


@pytest.mark.parametrize("where,want", [("grad_out", [1, 1, 0]), ("q", [1, 0, 1]), (None, [1, 0, 0])])
def test_two_products_from_one_plan(monkeypatch, where, want):
    """dV = P^T dO and dK = dS^T Q: an Inf in a row of dO, or of Q, whose vector-row has no keys makes a NaN of the densified sums of that
    product alone."""
    monkeypatch.setenv("VSPARSE_B200_SPMM_T", "dense")
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "fused")
    V, d, n = 8, 64, 160
    a = custom([0 if i == 5 else 24 for i in range(n // V)], n, V, seed=2)
    q, k, v, go = (cvse.fill_random((1, n, d), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0) for i in range(4))
    clean = [x[0].astype(np.float32) for x in (q, k, v, go)]
    if where:
        (go if where == "grad_out" else q)[0, 5 * V + 2, 9] = np.inf
    workspace = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV)
    gq, gk, gv = (torch.full((1, n, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(3))
    ws_p, ws_g = (torch.empty(a.nnz_vec * V, dtype=torch.float16, device=DEV) for _ in range(2))
    ops.set_workspace(workspace)
    try:
        ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *structure(a), *(dev(x) for x in cvse.transpose(a)), dev(q), dev(k),
                                    dev(v), dev(go), gq, gk, gv, ws_p, ws_g, 0.125)
        assert words(workspace) == want
    finally:
        ops.set_workspace(None)
    expected = oracle.attention_backward(a.m_vec, V, d, a.row_offsets, a.col_indices, *clean, 0.125)
    for got, w, what in zip((gq, gk, gv), expected, ("dQ", "dK", "dV")):
        assert_close(got[0].float().cpu().numpy(), w, what)
