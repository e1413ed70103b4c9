"""The one-kernel SpMM where several CTAs share a tile, each with a part of the matrix's columns: rows with all, no and one entry in a part, entries on both sides of
its ends, columns in another order or named twice within and across parts, non-finite operands, against the fp64 oracle."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from gpu_util import DEV, captured_kernels, custom, dev, spmm_oracle, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, ops, shard

pytestmark = pytest.mark.gpu


def matrix(V, K, m_vec, seed):
    rng = np.random.default_rng(seed)
    a = custom(np.resize([K, 0, 1, 40, 130, K // 2, 7, 300], m_vec), K, V, seed=seed)
    rows = [a.col_indices[a.row_offsets[i]:a.row_offsets[i + 1]] for i in range(m_vec)]   # views
    rows[4][:] = np.arange(130) + K - 130          # all in the last part
    rows[3][:] = np.arange(40)                     # all in the first one
    rows[7][:] = rng.permutation(rows[7])          # in another order
    rows[5][[0, -1]] = rows[5][[-1, 0]]            # two entries, parts apart
    rows[12][64] = rows[12][65]                    # a column named twice
    rows[13][-1] = rows[13][0]                     # in two places parts apart
    return a


@pytest.mark.parametrize("split", [2, 4, 8])
@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("K,N", [(3072, 72), (3073, 64), (3200, 8), (4095, 136)])
def test_shared_tiles(monkeypatch, V, K, N, split):
    monkeypatch.setenv("VSPARSE_B200_SPMM", "direct")
    monkeypatch.setenv("VSPARSE_B200_SPMM_SPLIT", str(split))
    a, batch = matrix(V, K, 21, V + K), 2
    rng = np.random.default_rng(K)
    row = (a.nnz_vec * V + 7) // 8 * 8
    # results of up to 0.05 sqrt(4095) x 6 = 19: rounding them to fp16 takes 2^-7 at most, the bound on the largest difference is 0.02
    vals, B = (0.05 * rng.standard_normal((batch, row))).astype(np.float16), rng.standard_normal((batch, K, N)).astype(np.float16)
    st = structure(a)
    for path, dtype in ((VS_PATH_CUDA_CORE, torch.float16),) if V == 1 or N % 64 else ((VS_PATH_CUDA_CORE, torch.float16), (VS_PATH_TENSOR, torch.float32)):
        out = torch.full((batch * a.m * N + 64,), float("nan"), dtype=dtype, device=DEV)
        operands = dev(vals), dev(B), out[:batch * a.m * N].view(batch, a.m, N)
        names = captured_kernels(lambda: ops.spmm_batched(path, a.m_vec, V, N, K, *st, *operands))
        torch.cuda.synchronize()
        assert ops.device_status() == 0 and "spmm_direct_kernel" in names and "Lb1E" in names
        assert bool(torch.isnan(out[batch * a.m * N:]).all())
        for b in range(batch):
            assert_close(operands[2][b].float().cpu().numpy(), spmm_oracle(a, N, vals[b, :a.nnz_vec * V], B[b]), f"entry {b}")


def test_non_finite_operands_and_parts_of_a_call(monkeypatch):
    V, K, N = 4, 3100, 192
    a = custom([K // 3] * 24, K, V, seed=3)
    rng = np.random.default_rng(1)
    vals, B = rng.standard_normal(a.nnz_vec * V).astype(np.float16), rng.standard_normal((K, N)).astype(np.float16)
    st, v = structure(a), dev(vals)

    def product(columns):
        rhs = dev(B[:, columns])
        out = torch.empty((a.m, rhs.shape[1]), dtype=torch.float32, device=DEV)
        ops.spmm.wmmaSpmm(a.m_vec, V, rhs.shape[1], K, *st, v, rhs, out)
        return out.cpu().numpy()
    whole = product(slice(None))
    with shard.part_of(columns=N):
        assert np.array_equal(product(slice(64, 128)), whole[:, 64:128])
    B[a.col_indices[5], 7] = np.inf
    got = product(slice(None))
    named = np.repeat([a.col_indices[5] in a.col_indices[a.row_offsets[i]:a.row_offsets[i + 1]] for i in range(a.m_vec)], V)
    assert 0 < named.sum() < a.m and not np.isfinite(got[named, 7]).any() and np.isfinite(got[~named]).all() and np.isfinite(np.delete(got, 7, 1)).all()
    want = spmm_oracle(a, N, vals, np.where(np.isfinite(B), B, 0))
    assert_close(np.delete(got, 7, 1), np.delete(want, 7, 1), "other columns")
    assert_close(got[~named, 7], want[~named, 7], "rows that do not name it")
