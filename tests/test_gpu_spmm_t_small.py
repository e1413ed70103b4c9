"""Small transposed products: one launch of the CUDA-core kernel, no plan; on either side of the line against the fp64 oracle."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, captured_kernels, custom, dev
from vectorsparse_b200 import cvse, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("m_vec,V,n,N,small", [(61, 4, 719, 520, True), (61, 4, 719, 576, False), (512, 2, 96, 64, True), (520, 2, 96, 64, False),
                                               (1, 8, 8, 8, True)])
def test_small_products_without_a_plan(monkeypatch, m_vec, V, n, N, small, dtype):
    """Up to 1e8 multiply-adds of a full matrix and 512 vector-rows one product goes to the CUDA-core kernel at once."""
    monkeypatch.delenv("VSPARSE_B200_SPMM_T", raising=False)
    a = custom([n // 2] * m_vec, n, V, seed=m_vec)
    t = [dev(x) for x in cvse.transpose(a)]
    vals = cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 3, 1.0)
    # sums of up to 512 products of standard deviation 1/4 stay below 4.5 * sqrt(512) / 4 < 32, where rounding to fp16 is at most 2^-7
    rhs = cvse.fill_random((a.m, N), np.float16, cvse.DIST_NORMAL, 4, 0.25)
    d_vals, d_rhs, out = dev(vals), dev(rhs), torch.full((n, N), float("nan"), dtype=dtype, device=DEV)
    names = captured_kernels(lambda: ops.spmm_t(a.m_vec, V, N, n, *t, d_vals, d_rhs, out, a.nnz_vec))
    assert ("dense_plan_kernel" not in names) == small and "spmm_t_kernel" in names, names
    want = oracle.spmm_t(a.m_vec, V, N, n, a.row_offsets, a.col_indices, vals.astype(np.float32), rhs.astype(np.float32))
    assert_close(out.float().cpu().numpy(), want, f"{m_vec} x {n} x {N}, V = {V}")
