"""The pair kernel at dense widths that are no multiple of 64: the bits of the single-CTA kernel, nothing past a row's end, for the product and its transpose, from a plan
and with the matrix laid out."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, captured_kernels, dev, problem, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, cvse, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("N", [136, 184, 200, 264, 312, 328, 392, 520])
@pytest.mark.parametrize("laid_out", ["plan", "laid-out"])
def test_product(monkeypatch, V, N, laid_out):
    monkeypatch.setenv("VSPARSE_B200_SPMM", "dense")
    monkeypatch.setenv("VSPARSE_B200_SPMM_A", laid_out)
    a = problem(cvse.GEN_BETA, 5, 300 // V, 333, V, 0.8)
    rng, batch = np.random.default_rng(N), 2
    row = (a.nnz_vec * V + 7) // 8 * 8
    st, vals, B = structure(a), dev(rng.standard_normal((batch, row)).astype(np.float16)), dev(rng.standard_normal((batch, a.n, N)).astype(np.float16))
    got = {}
    for pair in ("1", "0"):
        monkeypatch.setenv("VSPARSE_B200_SPMM_PAIR", pair)
        flat = torch.full((batch * a.m * N + 64,), float("nan"), dtype=torch.float16, device=DEV)
        out = flat[:batch * a.m * N].view(batch, a.m, N)
        names = captured_kernels(lambda: ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, V, N, a.n, *st, vals, B, out))
        torch.cuda.synchronize()
        assert ops.device_status() == 0 and bool(torch.isnan(flat[batch * a.m * N:]).all())
        assert ("spmm_pair_kernel" in names) == (pair == "1") and ("densify_kernel" in names) == (pair == "1" and V <= 2 and laid_out == "laid-out")
        got[pair] = out.cpu().numpy()
    assert np.array_equal(got["1"], got["0"])


@pytest.mark.parametrize("V", [2, 8])
@pytest.mark.parametrize("N", [136, 200, 264, 328])
def test_transposed_product(monkeypatch, V, N):
    monkeypatch.setenv("VSPARSE_B200_SPMM_T", "dense")
    a = problem(cvse.GEN_BETA, 7, 320 // V, 300, V, 0.7)
    rng = np.random.default_rng(N)
    t, vals, rhs = [dev(x) for x in cvse.transpose(a)], dev(rng.standard_normal(a.nnz_vec * V).astype(np.float16)), dev(rng.standard_normal((a.m, N)).astype(np.float16))
    got = {}
    for pair in ("1", "0"):
        monkeypatch.setenv("VSPARSE_B200_SPMM_PAIR", pair)
        flat = torch.full((a.n * N + 64,), float("nan"), dtype=torch.float16, device=DEV)
        out = flat[:a.n * N].view(a.n, N)
        names = captured_kernels(lambda: ops.spmm_t(a.m_vec, V, N, a.n, *t, vals, rhs, out, a.nnz_vec))
        torch.cuda.synchronize()
        assert ops.device_status() == 0 and bool(torch.isnan(flat[a.n * N:]).all()) and ("spmm_pair_kernel" in names) == (pair == "1")
        got[pair] = out.cpu().numpy()
    assert np.array_equal(got["1"], got["0"])
