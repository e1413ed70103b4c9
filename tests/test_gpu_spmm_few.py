"""CUDA-core SpMM for products that leave most of the GPU idle: every output once, with the bits of spmm_cc_kernel, whose sums are in the same order."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, captured_kernels, custom, dev, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, ops

pytestmark = pytest.mark.gpu
LENS = [0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 63, 64, 65, 96, 97, 130]   # on both sides of the entries in flight and of those passed round


def run(a, N, dtype, batch, out_dtype, seed=0):
    rng = np.random.default_rng(seed)
    row = (a.nnz_vec * a.V + 7) // 8 * 8
    vals, B = (rng.uniform(-1, 1, s).astype(dtype) for s in ((batch, row), (batch, a.n, N)))
    B[0, a.col_indices[20], N // 2] = np.inf
    B[-1, a.col_indices[5], 0] = np.nan
    vals, B, st = dev(vals), dev(B), structure(a)
    flat = torch.full((batch * a.m * N + 64,), float("nan"), dtype=out_dtype, device=DEV)
    out = flat[:batch * a.m * N].view(batch, a.m, N)

    def call():
        ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, a.V, N, a.n, *st, vals, B, out)
    call()
    torch.cuda.synchronize()
    assert bool(torch.isnan(flat[batch * a.m * N:]).all())
    return out.clone(), call


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("dtype,widths", [(np.float32, (4, 28, 32, 36, 132)), (np.float16, (8, 56, 64, 72, 264))])
def test_four_byte_lanes(monkeypatch, V, dtype, widths):
    monkeypatch.setenv("VSPARSE_B200_SPMM_F32", "cores")
    a = custom(LENS, 140, V, seed=V)
    rng = np.random.default_rng(V)
    a.col_indices[a.row_offsets[15]:a.row_offsets[16]] = rng.integers(0, 140, LENS[15])   # unsorted, some twice
    for N in widths:
        got = {}
        for mode in ("rows", "few", None):   # by itself as well: all of these are small
            monkeypatch.setenv("VSPARSE_B200_SPMM_CC", mode) if mode else monkeypatch.delenv("VSPARSE_B200_SPMM_CC")
            got[mode], call = run(a, N, dtype, 2, torch.float32)
            assert ("spmm_cc_few_kernel" in captured_kernels(call)) == (mode != "rows")
        assert torch.equal(got["rows"].nan_to_num(nan=7.0), got["few"].nan_to_num(nan=7.0)) and torch.equal(got["few"].nan_to_num(nan=7.0), got[None].nan_to_num(nan=7.0))


@pytest.mark.parametrize("dtype,N", [(np.float32, 264), (np.float16, 528)])
def test_sixteen_byte_lanes(monkeypatch, dtype, N):
    """V = 1 with more rows than 4-byte lanes are good for; the last piece of a row is partly empty."""
    monkeypatch.setenv("VSPARSE_B200_SPMM_F32", "cores")
    a = custom(np.resize(LENS, 1200), 140, 1)
    few, call = run(a, N, dtype, 1, torch.float32)
    assert "spmm_cc_few_kernel" in captured_kernels(call) and "Li1ELi16E" in captured_kernels(call)
    monkeypatch.setenv("VSPARSE_B200_SPMM_CC", "rows")
    rows, call = run(a, N, dtype, 1, torch.float32)
    assert "spmm_cc_few_kernel" not in captured_kernels(call)
    assert torch.equal(rows.nan_to_num(nan=7.0), few.nan_to_num(nan=7.0))
