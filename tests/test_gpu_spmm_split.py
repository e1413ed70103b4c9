"""fp32 SpMM from bf16 parts on the tensor cores, forced, against the fp64 oracle: no further from it than the CUDA-core kernel, and what it
hands to that kernel comes back with that kernel's bits."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, custom, dev, problem, spmm_oracle, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, cvse, ops

pytestmark = pytest.mark.gpu


def run(monkeypatch, a, N, vals, B, mode, batch=1):
    monkeypatch.setenv("VSPARSE_B200_SPMM_F32", mode)
    out = torch.full((batch * a.m * N + 64,), float("nan"), device=DEV)
    view = out[:batch * a.m * N].view(batch, a.m, N)
    ops.kernel_timing(True)
    if batch > 1:
        ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, a.V, N, a.n, *structure(a), dev(vals), dev(B), view)
    else:
        ops.spmm.cudaSpmm(a.m_vec, a.V, N, a.n, *structure(a), dev(vals), dev(B), view)
    assert ops.kernel_timing(False)[1] == (1 if mode == "split" else 0), "not the kernels this is about"
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert bool(torch.isnan(out[batch * a.m * N:]).all()), "wrote past the end"
    return view.cpu().numpy()


# rows around the pair's 256 and a CTA's 128, columns around the 64 of a stage and 8192 / V of a preparation step, dense widths around the
# 64 of the parts, the 128 and 256 of a tile
@pytest.mark.parametrize("V,m_vec,K,N", [(1, 1, 1, 4), (1, 257, 63, 260), (1, 300, 129, 508), (2, 129, 64, 128), (2, 64, 4160, 68), (4, 65, 200, 252),
                                         (8, 17, 1100, 1024), (8, 100, 65, 132)])
@pytest.mark.parametrize("sparsity", [0.0, 0.6])
def test_edges(monkeypatch, V, m_vec, K, N, sparsity):
    a = problem(cvse.GEN_UNIFORM, 3, m_vec, K, V, sparsity)
    rng = np.random.default_rng(K)
    vals = rng.uniform(-1, 1, max(a.nnz_vec, 1) * V).astype(np.float32)
    B = rng.standard_normal((K, N)).astype(np.float32)
    want = spmm_oracle(a, N, vals[:a.nnz_vec * V], B).reshape(a.m, N)
    # per 64 columns four truncations and one rounding of 2^-24 of a partial sum, random in sign from block to block: 5 x 65^0.5 x 2^-24 =
    # 2.4e-6 of one block's sum at K = 4160, an eighth of that of the whole
    got = run(monkeypatch, a, N, vals, B, "split")[0]
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want) + 1e-30


@pytest.mark.parametrize("V,K,sparsity", [(1, 4096, 0.5), (1, 1024, 0.8), (2, 2048, 0.7), (4, 4096, 0.5), (8, 512, 0.5)])
def test_no_further_from_the_exact_sums_than_the_cuda_core_kernel(monkeypatch, V, K, sparsity):
    a = problem(cvse.GEN_UNIFORM, 7, 512 // V, K, V, sparsity)
    rng = np.random.default_rng(V)
    vals = rng.uniform(-1, 1, a.nnz_vec * V).astype(np.float32)
    B = rng.uniform(-1, 1, (K, 256)).astype(np.float32)
    want = spmm_oracle(a, 256, vals, B).reshape(a.m, 256)
    err = {m: np.linalg.norm(run(monkeypatch, a, 256, vals, B, m)[0] - want) for m in ("split", "cores")}
    assert err["split"] <= err["cores"], err


def test_batches_with_shared_operands(monkeypatch):
    V, batch, N = 4, 3, 320
    a = problem(cvse.GEN_BETA, 9, 70, 150, V, 0.6)
    rng = np.random.default_rng(0)
    row = (a.nnz_vec * V + 7) // 8 * 8
    vals = rng.uniform(-1, 1, (batch, row)).astype(np.float32)
    B = rng.uniform(-1, 1, (batch, a.n, N)).astype(np.float32)
    for v, b in ((vals, B), (vals[0], B), (vals, B[0])):
        got = run(monkeypatch, a, N, v, b, "split", batch)
        for i in range(batch):
            want = spmm_oracle(a, N, (v[i] if v.ndim == 2 else v)[:a.nnz_vec * V], b[i] if b.ndim == 3 else b).reshape(a.m, N)
            assert np.linalg.norm(got[i] - want) <= 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("what", ["repeated", "inf value", "nan in B", "largest", "tiny value", "tiny in B", "tiny result"])
def test_what_the_split_product_leaves_to_the_cuda_core_kernel(monkeypatch, what):
    V, N = 2, 256
    a = custom([40] * 150, 200, V, seed=5)
    rng = np.random.default_rng(1)
    vals = rng.uniform(-1, 1, a.nnz_vec * V).astype(np.float32)
    B = rng.uniform(-1, 1, (a.n, N)).astype(np.float32)
    if what == "repeated":
        a.col_indices[40 * 7 + 11] = a.col_indices[40 * 7 + 10]
    elif what == "inf value":
        vals[77] = np.inf
    elif what == "nan in B":
        B[3, 250] = np.nan
    elif what == "largest":
        vals[5] = np.finfo(np.float32).max
    elif what == "tiny value":
        vals[9] = 1e-38
    elif what == "tiny in B":
        B[199, 0] = -1e-35
    else:
        vals *= 2.0 ** -60
        B *= 2.0 ** -50
    assert np.array_equal(run(monkeypatch, a, N, vals, B, "split"), run(monkeypatch, a, N, vals, B, "cores"), equal_nan=True)
