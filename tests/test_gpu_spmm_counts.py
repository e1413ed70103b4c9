"""Who decides between the tiles of the one-kernel SpMM and the gather kernel: the host by the number of values where a call says it (one problem), or where even the distance
between the matrices of a batch leaves too few; else the device, which knows the number, with the gather kernel standing by."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from gpu_util import captured_kernels, custom, dev, spmm_oracle, structure
from vectorsparse_b200 import VS_PATH_TENSOR, ops

pytestmark = pytest.mark.gpu


# 64 vector-rows x 1024 columns: 32 stages (of 256 rows and 64 columns) at 1100 against 370 a vector-row and 4.7 an entry put the line at 2451 vectors
@pytest.mark.parametrize("per_row,pitch,batch,tiles,gather", [(300, 1, 1, True, False), (20, 1, 1, False, True), (20, 1, 2, False, True), (300, 1, 2, True, True),
                                                              (20, 5, 2, True, True)])
def test_who_decides(monkeypatch, per_row, pitch, batch, tiles, gather):
    monkeypatch.delenv("VSPARSE_B200_SPMM", raising=False)
    V, m_vec, K, N = 8, 64, 1024, 64
    a = custom([per_row] * m_vec, K, V, seed=per_row)
    rng = np.random.default_rng(batch)
    # sums of up to 0.05 sqrt(300) x 6 = 5
    vals, B = (0.05 * rng.standard_normal((batch, pitch * a.nnz_vec * V))).astype(np.float16), rng.standard_normal((batch, K, N)).astype(np.float16)
    st, out = structure(a), torch.full((batch, a.m, N), float("nan"), device="cuda:0")
    operands = dev(vals), dev(B), out
    names = captured_kernels(lambda: ops.spmm_batched(VS_PATH_TENSOR, a.m_vec, V, N, K, *st, *operands))
    assert ("spmm_direct_kernel" in names, "spmm_tma_kernel" in names or "spmm_tc_kernel" in names) == (tiles, gather), names
    assert ops.device_status() == 0
    for b in range(batch):
        assert_close(out[b].cpu().numpy(), spmm_oracle(a, N, vals[b, :a.nnz_vec * V], B[b]), f"entry {b}")
