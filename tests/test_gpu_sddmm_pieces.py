"""CUDA-core SDDMM with fp32 results where several groups of lanes share a vector-row: every entry once, against the fp64 oracle, with the bits of a batch so large
that a row has one group."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, captured_kernels, custom, dev, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("k", [8, 64, 72, 136, 256])
@pytest.mark.parametrize("lens", [[0, 1, 2, 15, 16, 17, 63, 64, 65, 300], [1100, 0, 3], [33]])
def test_every_entry_once(V, k, lens):
    a = custom(lens, 1200, V, seed=V + k)
    rng = np.random.default_rng(k)
    lhs, rhs = (rng.standard_normal((rows, k)).astype(np.float16) for rows in (a.m, a.n))
    st, size = structure(a), (a.nnz_vec * V + 3) // 4 * 4

    def run(batch):
        out = torch.full((batch * size + 64,), float("nan"), device=DEV)
        operands = dev(lhs).expand(batch, -1, -1).contiguous(), dev(rhs).expand(batch, -1, -1).contiguous(), out[:batch * size].view(batch, size)
        names = captured_kernels(lambda: ops.sddmm_batched(VS_PATH_CUDA_CORE, a.m_vec, k, a.n, a.nnz_vec, *st, *operands, V))
        torch.cuda.synchronize()
        assert "sddmm_cc_row_kernel" in names and bool(torch.isnan(out[batch * size:]).all())
        return operands[2][:, :a.nnz_vec * V]
    got = run(1)
    assert_close(got[0].cpu().numpy(), oracle.sddmm(a.m_vec, k, V, a.row_offsets, a.col_indices, lhs.astype(np.float32), rhs.astype(np.float32), acc="f64"), "entries")
    many = run(4 * 16 * 148 * 4 // a.m_vec // 8)
    assert bool((many == got).all())
