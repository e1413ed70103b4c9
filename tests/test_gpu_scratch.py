"""Whose memory the library's plans live in: the caller's workspace is the tensor path's alone, and a
stream's buffer belongs to one call at a time."""
import threading

import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, dev, problem, spmm_oracle, structure
from vectorsparse_b200 import _lib, cvse, ops

pytestmark = pytest.mark.gpu


class Products:
    """One structure with an SpMM and an SDDMM on it, their operands and oracle results."""

    def __init__(self, V, m_vec, K, N, sparsity, seed=1, kind=cvse.GEN_UNIFORM):
        self.a = a = problem(kind, seed, m_vec, K, V, sparsity)
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


@pytest.mark.parametrize("names", [("cudaSpmm", "cudaSddmm"), ("wmmaSpmm", "wmmaSddmm")])
def test_host_threads_can_share_a_stream(names):
    """Each call plans, multiplies and cleans up in several launches: those of another thread's call must not come between them."""
    problems = [Products(8, 1200, 1024, 512, 0.9, seed, cvse.GEN_FIXED) for seed in (1, 5)]   # of one size, so that a plan that is mixed up stays in bounds
    assert problems[0].a.nnz_vec == problems[1].a.nnz_vec
    stream, failures = torch.cuda.Stream(), []
    torch.cuda.synchronize()

    def calls(p):
        try:
            with torch.cuda.stream(stream):
                for i in range(200):
                    p.spmm(getattr(ops.spmm, names[0]))
                    p.sddmm(getattr(ops.sddmm, names[1]))
                    if i % 50 == 49:   # given up while the other thread works with it
                        _lib.lib().vs_release_scratch(stream.cuda_stream, 0)
        except Exception as e:
            failures.append(e)

    for p in problems:
        p.poison()
    torch.cuda.synchronize()
    threads = [threading.Thread(target=calls, args=(p,)) for p in problems]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    for i, p in enumerate(problems):
        p.check(f"thread {i}")
