"""fp32 SpMM from bf16 parts, row by row: a matrix that takes the tensor cores as a whole, with rows of every length among its long ones.  Rows with
few entries have the bits of the CUDA-core kernel, the others are no further from 64-bit sums than that kernel's."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, custom, dev, structure
from vectorsparse_b200 import ops

pytestmark = pytest.mark.gpu


def run(monkeypatch, a, N, vals, B, mode):
    if mode == "auto":
        monkeypatch.delenv("VSPARSE_B200_SPMM_F32", raising=False)
    else:
        monkeypatch.setenv("VSPARSE_B200_SPMM_F32", mode)
    out = torch.full((a.m, N), float("nan"), device=DEV)
    ops.spmm.cudaSpmm(a.m_vec, a.V, N, a.n, *structure(a), vals, B, out)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    return out


@pytest.mark.parametrize("operands", ["both signs", "positive", "near 1"])
@pytest.mark.parametrize("V,m_vec,long", [(1, 1024, 400), (4, 512, 600)])
def test_rows_of_every_length(monkeypatch, V, m_vec, long, operands):
    K, N, few = 2048, 2048, 2048 // 64 + 16
    lens = np.full(m_vec, long)
    short = [0, 1, 2, 3, 8, 24, few - 1, few, few + 1, few + 20]
    lens[np.arange(8 * len(short)) * 5] = np.repeat(short, 8)
    a = custom(lens, K, V, seed=1)
    rng = np.random.default_rng(V)
    draw = {"both signs": lambda s: rng.uniform(-1, 1, s), "positive": lambda s: rng.uniform(0, 1, s), "near 1": lambda s: 1 + rng.uniform(0, 0.02, s)}[operands]
    vals, B = dev(draw(a.nnz_vec * V).astype(np.float32)), dev(draw((K, N)).astype(np.float32))
    dense = torch.zeros((a.m_vec, V, K), dtype=torch.float64, device=DEV)
    rows = torch.from_numpy(np.repeat(np.arange(a.m_vec), np.diff(a.row_offsets))).to(DEV)
    dense[rows, :, torch.from_numpy(a.col_indices.astype(np.int64)).to(DEV)] = vals.view(-1, V).double()
    want = (dense.view(a.m, K) @ B.double()).view(a.m_vec, V, N)
    got, cores = (run(monkeypatch, a, N, vals, B, m).view(a.m_vec, V, N) for m in ("auto", "cores"))
    at = torch.from_numpy(lens).to(DEV)
    assert torch.equal(got[at < few], cores[at < few])
    assert not torch.equal(got[at == long], cores[at == long]), "the tensor cores have not taken the product"
    for n in (few, few + 1, few + 20, long):
        err = [torch.linalg.norm(x[at == n].double() - want[at == n]).item() for x in (got, cores)]
        assert err[0] <= err[1], (n, err)
