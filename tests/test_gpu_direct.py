"""The one-kernel forms of the tensor-core products (small problems), forced at the sizes where their tiles, chunks and
windows end, and on the inputs they hand to their entry-by-entry path; against the fp64 oracle, conftest tolerance."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, custom, dev, problem, spmm_oracle, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, _lib, cvse, ops

pytestmark = pytest.mark.gpu


def spmm_forced(monkeypatch, a, N, vals, B, out_t, mode):
    monkeypatch.setenv("VSPARSE_B200_SPMM", mode)
    out = torch.full((a.m, N), float("nan"), dtype=out_t, device=DEV)
    ops.spmm.wmmaSpmm(a.m_vec, a.V, N, a.n, *structure(a), dev(vals), dev(B), out)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    return out.float().cpu().numpy()


# rows around the 128-row tile, columns around the 128-column chunk and the three-chunk ring, an empty matrix and full
# rows (a chunk holds more than two windows of a row)
@pytest.mark.parametrize("V,m_vec,K,N,sparsity", [(8, 1, 1, 64, 0.0), (8, 16, 128, 64, 0.5), (8, 17, 129, 128, 0.9), (8, 33, 700, 192, 0.95),
                                                  (4, 31, 127, 64, 0.0), (4, 33, 513, 64, 0.8), (2, 63, 64, 64, 0.7), (2, 65, 385, 128, 0.1),
                                                  (8, 20, 300, 64, 1.0)])
@pytest.mark.parametrize("out_t", [torch.float16, torch.float32])
def test_direct_spmm_at_the_edges_of_its_tiles(monkeypatch, V, m_vec, K, N, sparsity, out_t):
    a = problem(cvse.GEN_UNIFORM, 3, m_vec, K, V, sparsity)
    vals = cvse.fill_random((max(a.nnz_vec, 1) * V,), np.float16, cvse.DIST_NORMAL, 1, 0.25)
    B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 0.5)
    got = spmm_forced(monkeypatch, a, N, vals, B, out_t, "direct")
    assert_close(got, spmm_oracle(a, N, vals[:a.nnz_vec * V], B), "direct")
    if sparsity < 1.0:   # the same K order, so the same bits as the kernels that work from a plan
        assert np.array_equal(got, spmm_forced(monkeypatch, a, N, vals, B, out_t, "dense"))


@pytest.mark.parametrize("V", [2, 8])
@pytest.mark.parametrize("what", ["unsorted", "repeated", "non-finite"])
def test_direct_spmm_tiles_computed_entry_by_entry(monkeypatch, V, what):
    """Unsorted columns, a column named twice, and an Inf in a row of B that one vector-row names: only that row may
    become non-finite."""
    K, N = 200, 128
    a = custom([40] * (300 // V), K, V, seed=5)
    vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.25)
    B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 0.5)
    if what == "unsorted":
        ci = a.col_indices.reshape(-1, 40)
        ci[3] = ci[3, ::-1]
    elif what == "repeated":
        a.col_indices[40 * 7 + 11] = a.col_indices[40 * 7 + 10]
    else:
        B[a.col_indices[0], 5] = np.inf
    want = spmm_oracle(a, N, vals, B)
    got = spmm_forced(monkeypatch, a, N, vals, B, torch.float32, "direct")
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite)
    assert_close(got[finite], want[finite], what)


@pytest.mark.parametrize("V,m_vec,n,k,lens", [(8, 1, 1, 64, [1]), (8, 17, 129, 192, None), (4, 33, 63, 64, None), (2, 65, 257, 320, None),
                                              (8, 16, 2000, 64, [1500] * 16), (2, 64, 128, 128, [0, 128] * 32)])
@pytest.mark.parametrize("out_t", [torch.float16, torch.float32])
def test_direct_sddmm_at_the_edges_of_its_tiles(monkeypatch, V, m_vec, n, k, lens, out_t):
    """Rows around the 128-row tile, mask columns around the 64-column one, more contraction blocks than ring stages, rows with
    more entries than are looked up ahead, unsorted and repeated columns."""
    lens = lens or [(7 * i) % min(n, 40) for i in range(m_vec)]
    a = custom(lens, n, V, seed=9)
    rng = np.random.default_rng(1)
    if a.nnz_vec > 4:   # any order, any repetition
        first = slice(int(a.row_offsets[m_vec - 1]), int(a.row_offsets[m_vec]))
        a.col_indices[first] = rng.permutation(a.col_indices[first])
        a.col_indices[a.nnz_vec // 2] = a.col_indices[a.nnz_vec // 2 - 1]
    lhs = cvse.fill_random((a.m, k), np.float16, cvse.DIST_NORMAL, 3, 0.25)
    rhs = cvse.fill_random((n, k), np.float16, cvse.DIST_NORMAL, 4, 0.25)
    monkeypatch.setenv("VSPARSE_B200_SDDMM", "direct")
    out = torch.full((a.nnz_vec * V + 8,), float("nan"), dtype=out_t, device=DEV)
    ops._sddmm(VS_PATH_TENSOR, m_vec, k, n, a.nnz_vec, *structure(a), dev(lhs), dev(rhs), out, V, 1)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    want = oracle.sddmm(m_vec, k, V, a.row_offsets, a.col_indices, lhs.astype(np.float32), rhs.astype(np.float32), acc="f64")
    assert_close(out[:a.nnz_vec * V].float().cpu().numpy(), want, "direct")
    assert torch.isnan(out[a.nnz_vec * V:]).all()


@pytest.mark.parametrize("mode", ["direct", "dense", "gather"])
@pytest.mark.parametrize("V,m_vec,K,N", [(1, 130, 200, 72), (2, 70, 129, 136), (4, 40, 300, 8), (8, 33, 64, 264)])
def test_cuda_core_spmm_with_fp16_results_in_every_form(monkeypatch, mode, V, m_vec, K, N):
    """The entry point that takes V = 1 and dense widths that are multiples of 8: its one-kernel form, its planned form on single CTAs
    and the CUDA-core kernel; a column named twice on top of each."""
    monkeypatch.setenv("VSPARSE_B200_SPMM", mode)
    a = problem(cvse.GEN_BETA, 8, m_vec, K, V, 0.7)
    for repeat in (False, True):
        if repeat:
            j = int(a.row_offsets[np.argmax(np.diff(a.row_offsets))])
            a.col_indices[j + 1] = a.col_indices[j]
        vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.25)
        B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 0.5)
        out = torch.full((a.m, N), float("nan"), dtype=torch.float16, device=DEV)
        ops.spmm.cudaSpmm(m_vec, V, N, K, *structure(a), dev(vals), dev(B), out)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        assert_close(out.float().cpu().numpy(), spmm_oracle(a, N, vals, B), f"{mode}, repeated column: {repeat}")


@pytest.mark.parametrize("N", [128, 256])
@pytest.mark.parametrize("V,m_vec,K", [(1, 300, 200), (2, 130, 449), (4, 70, 300), (8, 33, 640)])
@pytest.mark.parametrize("what", ["plain", "repeated", "non-finite"])
def test_cuda_core_spmm_behind_the_pair_kernel(monkeypatch, V, m_vec, K, N, what):
    """Dense widths of the pair kernel, at every vector length; a column named twice, and an Inf in a row of B that some vector-rows name
    and others do not, send the call to the CUDA-core kernel behind it."""
    monkeypatch.setenv("VSPARSE_B200_SPMM", "dense")
    a = problem(cvse.GEN_BETA, 8, m_vec, K, V, 0.7)
    vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.25)
    B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 0.5)
    if what == "repeated":
        j = int(a.row_offsets[np.argmax(np.diff(a.row_offsets))])
        a.col_indices[j + 1] = a.col_indices[j]
    elif what == "non-finite":
        B[a.col_indices[0], 5] = np.inf
    out = torch.full((a.m, N), float("nan"), dtype=torch.float16, device=DEV)
    pairs = ctypes.c_int(0)
    _lib.lib().vs_kernel_timing(1, None, None)
    ops.spmm.cudaSpmm(m_vec, V, N, K, *structure(a), dev(vals), dev(B), out)
    _lib.lib().vs_kernel_timing(0, None, ctypes.byref(pairs))
    torch.cuda.synchronize()
    assert ops.device_status() == 0 and pairs.value == 1   # the pair kernels are the ones that are timed
    got, want = out.float().cpu().numpy(), spmm_oracle(a, N, vals, B)
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite) and finite.all() == (what != "non-finite")
    assert_close(got[finite], want[finite], what)


@pytest.mark.parametrize("V", [1, 2, 8])
def test_one_kernel_spmm_with_one_dense_operand_for_the_batch(monkeypatch, V):
    monkeypatch.setenv("VSPARSE_B200_SPMM", "direct")
    a = problem(cvse.GEN_UNIFORM, 4, 200 // V, 300, V, 0.8)
    row = (a.nnz_vec * V + 7) // 8 * 8
    vals = cvse.fill_random((3, row), np.float16, cvse.DIST_NORMAL, 1, 0.25)
    B = cvse.fill_random((300, 72), np.float16, cvse.DIST_NORMAL, 2, 0.5)
    out = torch.full((3, a.m, 72), float("nan"), dtype=torch.float16, device=DEV)
    ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, V, 72, 300, *structure(a), dev(vals), dev(B), out)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for b in range(3):
        assert_close(out[b].float().cpu().numpy(), spmm_oracle(a, 72, vals[b, :a.nnz_vec * V], B), f"entry {b}")


@pytest.mark.parametrize("mode", ["direct", "dense", "gather"])
@pytest.mark.parametrize("V,m_vec,n,k", [(1, 130, 130, 8), (2, 70, 257, 72), (4, 33, 100, 200), (8, 40, 300, 456)])
def test_cuda_core_sddmm_with_fp16_results_in_every_form(monkeypatch, mode, V, m_vec, n, k):
    """Contraction lengths that are multiples of 8 and not of 64: the last block of the tiles is filled up with zeros."""
    monkeypatch.setenv("VSPARSE_B200_SDDMM", mode)
    a = problem(cvse.GEN_BETA, 8, m_vec, n, V, 0.7)
    lhs = cvse.fill_random((2, a.m, k), np.float16, cvse.DIST_NORMAL, 3, 0.25)
    rhs = cvse.fill_random((2, n, k), np.float16, cvse.DIST_NORMAL, 4, 0.25)
    row = (a.nnz_vec * V + 7) // 8 * 8
    out = torch.full((2, row), float("nan"), dtype=torch.float16, device=DEV)
    ops.sddmm_batched(VS_PATH_CUDA_CORE, m_vec, k, n, a.nnz_vec, *structure(a), dev(lhs), dev(rhs), out, V)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for b in range(2):
        want = oracle.sddmm(m_vec, k, V, a.row_offsets, a.col_indices, lhs[b].astype(np.float32), rhs[b].astype(np.float32), acc="f64")
        assert_close(out[b, :a.nnz_vec * V].float().cpu().numpy(), want, f"{mode}, entry {b}")


# rows around the 16 of a CTA, columns around the 128 of a tile and the three-tile ring, dense widths around the 128-column slab, full
# rows (more than one batch of entries per tile), rows with few entries (gathered instead of staged) and an empty matrix
@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("m_vec,K,N,sparsity", [(1, 1, 4, 0.0), (16, 128, 128, 0.0), (17, 129, 132, 0.5), (33, 513, 260, 0.3), (40, 700, 124, 0.97),
                                                (20, 640, 64, 1.0)])
@pytest.mark.parametrize("order", ["ascending", "mixed"])
def test_fp32_spmm_on_staged_tiles(monkeypatch, V, m_vec, K, N, sparsity, order):
    """The same bits as the kernel without staged tiles, whose sums are formed in the same order, and the oracle's values."""
    a = problem(cvse.GEN_UNIFORM, 3, m_vec, K, V, sparsity)
    if order == "mixed":   # every other row in any order, one of them with a column named twice
        rng = np.random.default_rng(1)
        for r in range(0, m_vec, 2):
            part = slice(int(a.row_offsets[r]), int(a.row_offsets[r + 1]))
            a.col_indices[part] = rng.permutation(a.col_indices[part])
        if a.row_offsets[1] > 1:
            a.col_indices[1] = a.col_indices[0]
    row = (max(a.nnz_vec, 1) * V + 3) // 4 * 4
    vals = cvse.fill_random((2, row), np.float32, cvse.DIST_UNIFORM, 1)
    B = cvse.fill_random((2, K, N), np.float32, cvse.DIST_UNIFORM, 2)
    got = {}
    for mode in ("rows", "tiles"):
        monkeypatch.setenv("VSPARSE_B200_SPMM_CC", mode)
        out = torch.full((2, a.m, N), float("nan"), dtype=torch.float32, device=DEV)
        ops.spmm_batched(VS_PATH_CUDA_CORE, m_vec, V, N, K, *structure(a), dev(vals), dev(B), out)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        got[mode] = out.cpu().numpy()
    assert np.array_equal(got["rows"], got["tiles"])
    for b in range(2):
        assert_close(got["tiles"][b], spmm_oracle(a, N, vals[b, :a.nnz_vec * V], B[b]), f"entry {b}")


@pytest.mark.parametrize("shared", [False, True])
def test_fp32_spmm_on_staged_tiles_with_non_finite_operands(monkeypatch, shared):
    """Inf and NaN reach the rows that name them and no others; one dense operand for the whole batch."""
    a = problem(cvse.GEN_UNIFORM, 4, 20, 200, 4, 0.5)
    row = (a.nnz_vec * 4 + 3) // 4 * 4
    vals = dev(cvse.fill_random((2, row), np.float32, cvse.DIST_UNIFORM, 1))
    B = cvse.fill_random((1 if shared else 2, 200, 132), np.float32, cvse.DIST_UNIFORM, 2)
    B[0, a.col_indices[0], 3] = np.inf
    B[0, a.col_indices[1], 130] = np.nan
    rhs = dev(B[0]) if shared else dev(B)
    got = {}
    for mode in ("rows", "tiles"):
        monkeypatch.setenv("VSPARSE_B200_SPMM_CC", mode)
        out = torch.zeros((2, a.m, 132), dtype=torch.float32, device=DEV)
        ops.spmm_batched(VS_PATH_CUDA_CORE, 20, 4, 132, 200, *structure(a), vals, rhs, out)
        torch.cuda.synchronize()
        got[mode] = out.cpu().numpy()
    assert not np.isfinite(got["rows"]).all()
    assert np.array_equal(got["rows"], got["tiles"], equal_nan=True)


# far from the line on either side
@pytest.mark.parametrize("V,m_vec,K,sparsity,route", [(1, 200, 1100, 0.99, "gather"), (1, 200, 1100, 0.7, "direct"), (2, 90, 1300, 0.99, "gather"),
                                                      (2, 90, 1300, 0.8, "direct"), (1, 1040, 1025, 0.995, "gather"), (8, 24, 4200, 0.997, "gather"), (8, 24, 4200, 0.9, "direct")])
def test_cuda_core_spmm_chooses_by_density(monkeypatch, V, m_vec, K, sparsity, route):
    """The device takes the one-kernel form or the CUDA-core kernel behind it, on either side of its line: the bits are those of the form that
    the line names and not of the other, whose sums are in another order."""
    N = 200
    a = problem(cvse.GEN_BETA, 8, m_vec, K, V, sparsity)
    vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.25)
    B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 3, 0.5)
    got = {}
    for mode in (None, "direct", "gather"):
        monkeypatch.setenv("VSPARSE_B200_SPMM", mode) if mode else monkeypatch.delenv("VSPARSE_B200_SPMM", raising=False)
        out = torch.full((a.m, N), float("nan"), dtype=torch.float16, device=DEV)
        ops.spmm.cudaSpmm(m_vec, V, N, K, *structure(a), dev(vals), dev(B), out)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        got[mode] = out.float().cpu().numpy()
    assert_close(got[None], spmm_oracle(a, N, vals, B), route)
    assert not np.array_equal(got["direct"], got["gather"])
    assert np.array_equal(got[None], got[route])


@pytest.mark.parametrize("V,m_vec,K,N", [(1, 600, 2100, 512), (1, 300, 1200, 64), (8, 128, 8300, 128)])
def test_cuda_core_products_in_a_graph(V, m_vec, K, N):
    """Captured on a stream that has made no call yet, replayed twice with other values, then called on that stream: sizes of the planned,
    the density-dependent and the pair form, which keep scratch outside a graph."""
    a = problem(cvse.GEN_UNIFORM, 3, m_vec, K, V, 0.9)
    st = structure(a)
    vals = [cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, seed, 0.25) for seed in (1, 2, 3)]
    B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 4, 0.5)
    lhs = cvse.fill_random((a.m, N), np.float16, cvse.DIST_NORMAL, 5, 0.25)
    v, b, l = dev(vals[0]), dev(B), dev(lhs)
    out = torch.empty((a.m, N), dtype=torch.float16, device=DEV)
    sampled = torch.empty((a.nnz_vec * V,), dtype=torch.float16, device=DEV)

    def products():
        ops.spmm.cudaSpmm(m_vec, V, N, K, *st, v, b, out)
        ops.sddmm.cudaSddmm(m_vec, N, K, a.nnz_vec, *st, l, b, sampled, V)

    def check(values, what):
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        assert_close(out.float().cpu().numpy(), spmm_oracle(a, N, values, B), what)
        want = oracle.sddmm(m_vec, N, V, a.row_offsets, a.col_indices, lhs.astype(np.float32), B.astype(np.float32), acc="f64")
        got = sampled.float().cpu().numpy()
        assert np.linalg.norm(got - want) <= 2e-3 * np.linalg.norm(want)   # fp16 results, 2^-11 each

    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        products()
    for values in vals[:2]:
        v.copy_(dev(values))
        out.fill_(float("nan"))
        sampled.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        check(values, "replay")
    v.copy_(dev(vals[2]))
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        products()
    check(vals[2], "after the graph")


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("N", [64, 72])
def test_direct_spmm_computes_only_the_odd_rows_entry_by_entry(monkeypatch, V, N):
    """A tile with columns in any order, columns named twice, columns outside the matrix and a non-finite sum, each in some of its
    vector-rows, which hold more entries than the lanes of a row fetch at a time, or none: the other rows keep their bits."""
    K = 300
    a = custom([70, 0, 33, 100, 1] * (180 // V // 5 + 1), K, V, seed=5)
    rows = lambda i: slice(int(a.row_offsets[i]), int(a.row_offsets[i + 1]))
    vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.25)
    B = cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 0.5)
    monkeypatch.setenv("VSPARSE_B200_SPMM", "direct")

    def product(ci, B):
        st = structure(a)
        out = torch.full((a.m, N), float("nan"), dtype=torch.float16, device=DEV)
        ops.spmm.cudaSpmm(a.m_vec, V, N, K, st[0], st[1], dev(ci), dev(vals), dev(B), out)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        return out.float().cpu().numpy()

    plain = product(a.col_indices, B)
    ci = a.col_indices.copy()
    ci[rows(0)] = ci[rows(0)][::-1]
    ci[rows(7)] = np.random.default_rng(1).permutation(ci[rows(7)])
    ci[rows(13)][40] = ci[rows(13)][39]
    ci[rows(12)][-1] = K + 5
    ci[rows(5)][0] = -3
    odd = [0, 7, 13, 12, 5]
    entries = vals.astype(np.float32).reshape(-1, V).copy()
    entries[(ci < 0) | (ci >= K)] = 0   # no entries
    a2 = cvse.CVSE(a.m_vec, K, V, a.row_offsets, np.clip(ci, 0, K - 1), a.row_indices)
    want = spmm_oracle(a2, N, entries.ravel(), B)
    got = product(ci, B)
    assert_close(got, want, "odd rows")
    untouched = np.repeat(~np.isin(np.arange(a.m_vec), odd), V)
    assert np.array_equal(got[untouched], plain[untouched])
    B[ci[rows(3)][50], 5] = np.inf   # named by some rows
    got, want = product(a.col_indices, B), spmm_oracle(a, N, vals, B)
    assert np.array_equal(np.isfinite(got), np.isfinite(want)) and not np.isfinite(want).all()
    assert np.array_equal(got[:, :5], plain[:, :5]) or np.allclose(got[:, :5], plain[:, :5], rtol=2e-3, atol=2e-3)
    assert_close(got[np.isfinite(want)], want[np.isfinite(want)], "non-finite operand")


@pytest.mark.parametrize("V,m,n,k,density", [(1, 4096, 4096, 128, 0.003), (2, 4096, 4096, 256, 0.001), (4, 4096, 4096, 128, 0.003), (8, 4096, 4096, 256, 0.01),
                                             (8, 512, 512, 1504, 0.3), (8, 16384, 16384, 64, 0.001)])
def test_cuda_core_sddmm_of_sparse_masks_keeps_to_the_cuda_cores(monkeypatch, V, m, n, k, density):
    """A few entries per row: the CUDA-core kernel's bits and not those of the tiles; a denser mask the other way round (0.3)."""
    a = custom([int(n * density)] * (m // V), n, V, seed=3)
    lhs = dev(cvse.fill_random((m, k), np.float16, cvse.DIST_NORMAL, 3, 0.25))
    rhs = dev(cvse.fill_random((n, k), np.float16, cvse.DIST_NORMAL, 4, 0.25))
    st, got = structure(a), {}
    for mode in (None, "direct", "gather"):
        monkeypatch.setenv("VSPARSE_B200_SDDMM", mode) if mode else monkeypatch.delenv("VSPARSE_B200_SDDMM", raising=False)
        got[mode] = torch.full((a.nnz_vec * V,), float("nan"), dtype=torch.float16, device=DEV)
        ops.sddmm.cudaSddmm(a.m_vec, k, n, a.nnz_vec, *st, lhs, rhs, got[mode], V)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(got[None], got["gather" if density < 0.1 else "direct"])
    assert density < 0.1 or not torch.equal(got["direct"], got["gather"])
    assert torch.allclose(got["direct"].float(), got["gather"].float(), rtol=2e-3, atol=2e-3 * 0.25 * 0.25 * k**0.5)
