"""Whose memory the library's plans live in: the caller's workspace is the tensor path's alone, and a
stream's buffer belongs to one call at a time, and a graph's to the graph."""
import ctypes
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


def captured(stream, *calls):
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        for call in calls:
            call()
    return graph


@pytest.mark.parametrize("warm", [False, True])
def test_a_graph_keeps_its_scratch(warm):
    """Products with a plan, captured on a stream with and without earlier calls; a larger call on that stream, then replays beside calls there."""
    small, large = Products(8, 1200, 1024, 512, 0.9), Products(8, 2500, 2048, 256, 0.9, 4)
    a = small.a
    transposed = [dev(x) for x in cvse.transpose(a)]
    out_t = torch.empty((a.n, small.N), dtype=torch.float16, device=DEV)
    want_t = oracle.spmm_t(a.m_vec, a.V, small.N, a.n, a.row_offsets, a.col_indices, small.vals.float().cpu().numpy(),
                           small.lhs.float().cpu().numpy())

    def products():
        small.spmm(ops.spmm.wmmaSpmm)
        small.sddmm(ops.sddmm.wmmaSddmm)
        ops.spmm_t(a.m_vec, a.V, small.N, a.n, *transposed, small.vals, small.lhs, out_t)

    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    if warm:
        with torch.cuda.stream(stream):
            products()
    graph = captured(stream, products)
    with torch.cuda.stream(stream):
        large.spmm(ops.spmm.wmmaSpmm)   # grows the stream's buffer
    torch.cuda.synchronize()
    for i in range(3):
        small.poison()
        out_t.fill_(float("nan"))
        large.poison()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            graph.replay()
        with torch.cuda.stream(stream):   # beside the replay
            large.spmm(ops.spmm.wmmaSpmm)
            large.sddmm(ops.sddmm.wmmaSddmm)
        small.check(f"replay {i}")
        large.check(f"beside replay {i}")
        assert_close(out_t.float().cpu().numpy(), want_t, f"transposed, replay {i}")


def test_graphs_give_their_scratch_back():
    """Captured again and again: what an earlier graph held serves a later one."""
    p, stream = Products(8, 1200, 2048, 512, 0.9), torch.cuda.Stream()   # a plan of 20 MB
    free = []
    for _ in range(12):
        graph = captured(stream, lambda: p.spmm(ops.spmm.wmmaSpmm))
        graph.replay()
        torch.cuda.synchronize()
        del graph
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    p.sddmm(ops.sddmm.wmmaSddmm)
    p.check("after the graphs")
    assert free[1] - free[-1] < 64 << 20
    assert _lib.lib().vs_release_scratch(stream.cuda_stream, 0) == 0


def test_a_workspace_of_the_stated_size_serves_the_pair_kernel():
    """A mask of 3 % of the vectors: the plan of the pair kernel is larger than that of the single-CTA kernel."""
    p = Products(8, 1200, 1024, 512, 0.97)
    size = _lib.lib().vs_sddmm_workspace_bytes(p.a.m_vec, p.a.n, p.a.nnz_vec)
    workspace = torch.full((size + 256,), 0x5A, dtype=torch.uint8, device=DEV)
    p.spmm(ops.spmm.wmmaSpmm)
    p.sampled.fill_(float("nan"))
    pairs = ctypes.c_int(0)
    ops.set_workspace(workspace[:size])
    _lib.lib().vs_kernel_timing(1, None, None)
    try:
        p.sddmm(ops.sddmm.wmmaSddmm)
    finally:
        _lib.lib().vs_kernel_timing(0, None, ctypes.byref(pairs))
        ops.set_workspace(None)
    p.check("in a workspace of that size")
    assert pairs.value == 1   # the pair kernels are the ones that are timed
    assert bool((workspace[size:] == 0x5A).all())


def test_a_large_plan_takes_about_what_it_needs():
    """4096 x 4096 at V = 1: 134 MB of entries."""
    p, stream = Products(1, 4096, 4096, 1024, 0.95), torch.cuda.Stream()
    torch.cuda.synchronize()
    _lib.lib().vs_release_scratch(None, 1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with torch.cuda.stream(stream):
        p.spmm(ops.spmm.cudaSpmm)
        p.sddmm(ops.sddmm.cudaSddmm)
    p.check("with a plan of its own")
    assert before - torch.cuda.mem_get_info()[0] < 200 << 20
    assert _lib.lib().vs_release_scratch(stream.cuda_stream, 0) == 0
