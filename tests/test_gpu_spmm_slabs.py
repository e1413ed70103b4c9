"""The order in which the fp32 CUDA-core SpMM takes its outputs changes with 4096 dense columns and 16384 warps (slab by slab): every output is written once, at
sizes on both sides of the line and widths whose pieces do and do not come in warps, with the bits of the narrow products."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, custom, dev, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("N", [4092, 4096, 4100, 4224, 4352, 4608, 8192])
@pytest.mark.parametrize("batch,m_vec", [(1, 2048), (2, 2047), (2, 600)])
def test_every_output_once(monkeypatch, V, N, batch, m_vec):
    monkeypatch.setenv("VSPARSE_B200_SPMM_F32", "cores")
    monkeypatch.setenv("VSPARSE_B200_SPMM_CC", "rows")
    a = custom(np.resize([0, 5, 70, 1, 33, 2, 9], m_vec if V < 8 else m_vec // 2), 90, V, seed=V)
    rng = np.random.default_rng(N)
    row = (a.nnz_vec * V + 7) // 8 * 8
    vals, B = dev(rng.uniform(-1, 1, (batch, row)).astype(np.float32)), torch.rand((batch, a.n, N), device=DEV) - 0.5
    out = torch.full((batch * a.m * N + 64,), float("nan"), device=DEV)
    view = out[:batch * a.m * N].view(batch, a.m, N)
    ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, V, N, a.n, *structure(a), vals, B, view)
    torch.cuda.synchronize()
    assert bool(torch.isnan(out[batch * a.m * N:]).all())
    for c in range(0, N, 1024):
        w = min(1024, N - c)
        part = torch.empty((batch, a.m, w), device=DEV)
        ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, V, w, a.n, *structure(a), vals, B[:, :, c:c + w].contiguous(), part)
        assert torch.equal(part, view[:, :, c:c + w])
