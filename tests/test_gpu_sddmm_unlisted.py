"""Sampled products whose caller counts more entries than the offsets list (a padded index array), with a column named twice in the last row: what the rows list is computed,
what stands behind them is not looked up."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, captured_kernels, custom, dev, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, cvse, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("lens", [[5, 0, 40], [300, 7, 250]])
def test_entries_behind_the_last_row(monkeypatch, V, lens):
    monkeypatch.setenv("VSPARSE_B200_SDDMM", "dense")
    n, k, extra = 320, 64, 100
    a = custom(lens, n, V, seed=V)
    last = a.col_indices[a.row_offsets[-2]:]   # a view
    last[-1] = last[0]
    free = np.setdiff1d(np.arange(n), last)   # columns that the last row does not name
    padded = cvse.CVSE(a.m_vec, n, V, a.row_offsets, np.concatenate([a.col_indices, np.resize(free, extra)]).astype(np.int32), a.row_indices)
    # operands of their own seeds: sums of 64 products of standard deviation 1/16 stay below 16 sqrt(64) / 16 = 8, where rounding to fp16 is at most 2^-9; unrelated
    # to one another, unlike two operands of one seed, whose equal rows sum up to 100 and round by 2^-5, more than the 0.02 allowed
    lhs, rhs = (cvse.fill_random((rows, k), np.float16, cvse.DIST_NORMAL, rows, 0.25) for rows in (a.m, n + 1000))
    rhs = rhs[:n]
    listed, counted = a.nnz_vec * V, (a.nnz_vec + extra) * V
    out = torch.full((counted,), float("nan"), dtype=torch.float16, device=DEV)
    st, operands = structure(padded), (dev(lhs), dev(rhs), out)
    names = captured_kernels(lambda: ops.sddmm.cudaSddmm(a.m_vec, k, n, a.nnz_vec + extra, *st, *operands, V))
    assert ops.device_status() == 0 and "sddmm_twin_kernel" in names
    want = oracle.sddmm(a.m_vec, k, V, a.row_offsets, a.col_indices, lhs.astype(np.float32), rhs.astype(np.float32), acc="f64")
    assert_close(out[:listed].float().cpu().numpy(), want, f"V = {V}")
    assert bool(torch.isnan(out[listed:]).all())
