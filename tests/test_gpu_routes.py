"""Which kernels a call takes when nothing forces them, on both sides of the lines, and the scratch-keeping forms under capture, on two streams and from
two threads."""
import threading

import numpy as np
import pytest
import torch

from gpu_util import DEV, captured_kernels, dev, problem, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu


class Product:
    def __init__(self, V, M, K, N, sparsity, dtype, seed=3, batch=1, extra=0):
        self.a = problem(cvse.GEN_UNIFORM, seed, M // V, K, V, sparsity)
        self.st, self.N, self.batch = structure(self.a), N, batch
        row = (self.a.nnz_vec * V + 7) // 8 * 8
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        lead = (batch,) if batch > 1 else ()
        draw = lambda *shape: (torch.rand(lead + shape, generator=gen, device=DEV) * 2 - 1).to(dtype)
        self.vals, self.B = draw(row + extra), draw(K, N)
        self.out = torch.full(lead + (self.a.m, N), float("nan"), dtype=dtype, device=DEV)
        dense = torch.zeros((batch, self.a.m_vec, V, K), dtype=torch.float64, device=DEV)
        rows = torch.from_numpy(np.repeat(np.arange(self.a.m_vec), np.diff(self.a.row_offsets))).to(DEV)
        cols = torch.from_numpy(self.a.col_indices.astype(np.int64)).to(DEV)
        for b in range(batch):
            vals = self.vals[b] if batch > 1 else self.vals
            dense[b][rows, :, cols] = vals[:self.a.nnz_vec * V].view(-1, V).double()
        self.want = (dense.view(batch, self.a.m, K) @ self.B.double().view(batch, K, N)).view(self.out.shape)
        self.tolerance = 2e-3 if dtype == torch.float16 else 1e-6

    def call(self):
        a = self.a
        if self.batch > 1:
            ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, a.V, self.N, a.n, *self.st, self.vals, self.B, self.out)
        else:
            ops.spmm.cudaSpmm(a.m_vec, a.V, self.N, a.n, *self.st, self.vals, self.B, self.out)

    def check(self, what=""):
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        err = torch.linalg.norm(self.out.double() - self.want) / torch.linalg.norm(self.want)
        assert err.item() <= self.tolerance, (what, err.item())
        self.out.fill_(float("nan"))


# the densities at which the CUDA cores keep every width, the cost line and the narrowest width; the tile kernel's products
@pytest.mark.parametrize("V,M,K,N,sparsity,batch,split", [
    (1, 2048, 2048, 1024, 0.80, 1, True), (1, 2048, 2048, 1024, 0.91, 1, False), (1, 2048, 2048, 252, 0.5, 1, False), (4, 2048, 2048, 2048, 0.75, 1, True),
    (4, 2048, 2048, 2048, 0.81, 1, False), (8, 2048, 1024, 1024, 0.5, 1, True), (8, 2048, 1024, 1024, 0.9, 1, False), (2, 1024, 256, 1024, 0.75, 8, True),
    (2, 1024, 256, 1024, 0.93, 8, False), (1, 512, 512, 512, 0.5, 1, False), (8, 2048, 4096, 1024, 0.82, 1, False)])
def test_fp32_products(V, M, K, N, sparsity, batch, split):
    p = Product(V, M, K, N, sparsity, torch.float32, batch=batch)
    p.call()
    p.check("called")
    kernels = captured_kernels(p.call)
    assert ("spmm_split_kernel" in kernels) == split
    p.check("replayed")


def test_more_values_declared_than_there_are():
    """The binding takes the length of `values` for their number; the device finds a tenth of them and leaves the call to the CUDA cores."""
    p = Product(1, 2048, 2048, 1024, 0.97, torch.float32, extra=1 << 20)
    assert "spmm_split_kernel" in captured_kernels(p.call)
    p.call()
    got = p.out.clone()
    p.check()
    short = p.vals[:(p.a.nnz_vec + 7) // 8 * 8].clone()
    out = torch.empty_like(got)
    ops.spmm.cudaSpmm(p.a.m_vec, 1, p.N, p.a.n, *p.st, short, p.B, out)
    assert torch.equal(out, got)


@pytest.mark.parametrize("V,M,K,N,sparsity,laid_out", [(1, 4096, 2048, 1024, 0.8, True), (1, 1024, 1024, 256, 0.8, False), (2, 4096, 4096, 1984, 0.7, True)])
def test_fp16_products(V, M, K, N, sparsity, laid_out):
    p = Product(V, M, K, N, sparsity, torch.float16)
    p.call()
    p.check("called")
    assert ("densify_kernel" in captured_kernels(p.call)) == laid_out
    p.check("replayed")


KEEPS_SCRATCH = [(1, 2048, 2048, 1024, 0.8, torch.float32, "spmm_split_kernel"), (1, 4096, 2048, 1024, 0.8, torch.float16, "densify_kernel")]


@pytest.mark.parametrize("shape", KEEPS_SCRATCH)
def test_replays_beside_larger_calls_on_the_stream_that_was_captured(shape):
    V, M, K, N, sparsity, dtype, kernel = shape
    p, large = Product(V, M, K, N, sparsity, dtype), Product(V, M + 1024, K + 1024, N, sparsity, dtype, seed=4)
    assert kernel in captured_kernels(p.call)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        p.call()
    for i in range(3):
        p.out.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            graph.replay()
        with torch.cuda.stream(stream):
            large.call()
        p.check(f"replay {i}")
        large.check(f"beside replay {i}")


@pytest.mark.parametrize("shape", KEEPS_SCRATCH)
@pytest.mark.parametrize("threads", [False, True])
def test_two_streams(shape, threads):
    V, M, K, N, sparsity, dtype, _ = shape
    problems = [Product(V, M, K, N, sparsity, dtype, seed) for seed in (3, 5)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    failures = []

    def calls(i, times):
        try:
            with torch.cuda.stream(streams[i]):
                for _ in range(times):
                    problems[i].call()
        except Exception as e:
            failures.append(e)

    if threads:
        workers = [threading.Thread(target=calls, args=(i, 40)) for i in range(2)]
        for w in workers:
            w.start()
        for w in workers:
            w.join()
    else:
        for _ in range(40):
            calls(0, 1)
            calls(1, 1)
    assert not failures
    for i, p in enumerate(problems):
        p.check(f"problem {i}")


@pytest.mark.parametrize("shape", KEEPS_SCRATCH)
def test_two_threads_on_one_stream(shape):
    V, M, K, N, sparsity, dtype, _ = shape
    problems = [Product(V, M, K, N, sparsity, dtype, seed) for seed in (3, 5)]
    stream, failures = torch.cuda.Stream(), []
    torch.cuda.synchronize()

    def calls(p):
        try:
            with torch.cuda.stream(stream):
                for _ in range(40):
                    p.call()
        except Exception as e:
            failures.append(e)

    workers = [threading.Thread(target=calls, args=(p,)) for p in problems]
    for w in workers:
        w.start()
    for w in workers:
        w.join()
    assert not failures
    for i, p in enumerate(problems):
        p.check(f"thread {i}")
