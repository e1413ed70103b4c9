"""Whose memory the library's plans live in: the caller's workspace is the tensor path's alone."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, dev, problem, spmm_oracle, structure
from vectorsparse_b200 import cvse, ops

pytestmark = pytest.mark.gpu


class Products:
    """One structure with an SpMM and an SDDMM on it, their operands and oracle results."""

    def __init__(self, V, m_vec, K, N, sparsity, seed=1):
        self.a = a = problem(cvse.GEN_UNIFORM, seed, m_vec, K, V, sparsity)
        self.st, self.N = structure(a), N
        vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, seed, 0.25)
        B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, seed + 1, 0.25)
        lhs = cvse.fill_random((a.m, N), np.float16, cvse.DIST_NORMAL, seed + 2, 0.25)
        self.vals, self.B, self.lhs = dev(vals), dev(B), dev(lhs)
        self.c = torch.empty((a.m, N), dtype=torch.float16, device=DEV)
        self.sampled = torch.empty((a.nnz_vec * V,), dtype=torch.float16, device=DEV)
        self.want_c = spmm_oracle(a, N, vals, B)
        self.want_s = oracle.sddmm(a.m_vec, N, V, a.row_offsets, a.col_indices, lhs.astype(np.float32), B.astype(np.float32), acc="f64")

    def spmm(self, f):
        f(self.a.m_vec, self.a.V, self.N, self.a.n, *self.st, self.vals, self.B, self.c)

    def sddmm(self, f):
        f(self.a.m_vec, self.N, self.a.n, self.a.nnz_vec, *self.st, self.lhs, self.B, self.sampled, self.a.V)

    def poison(self):
        self.c.fill_(float("nan"))
        self.sampled.fill_(float("nan"))

    def check(self, what):
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        assert_close(self.c.float().cpu().numpy(), self.want_c, what + ": product")
        assert_close(self.sampled.float().cpu().numpy(), self.want_s, what + ": sampled")


@pytest.mark.parametrize("V,m_vec", [(1, 2400), (8, 1200)])
def test_cuda_core_calls_leave_the_callers_workspace_alone(V, m_vec):
    """A thread that set a workspace for its tensor-path calls may make cuda* calls on other streams beside them: sizes whose plans would
    live there."""
    p = Products(V, m_vec, 2100, 512, 0.8)
    workspace = torch.full((64 << 20,), 0x5A, dtype=torch.uint8, device=DEV)
    ops.set_workspace(workspace)
    try:
        p.poison()
        p.spmm(ops.spmm.cudaSpmm)
        p.sddmm(ops.sddmm.cudaSddmm)
        p.check("with a workspace")
    finally:
        ops.set_workspace(None)
    assert bool((workspace == 0x5A).all())
