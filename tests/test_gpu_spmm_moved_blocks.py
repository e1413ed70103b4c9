"""The one-kernel SpMM where several CTAs share a tile, on rows whose columns ascend in long runs but not throughout: blocks of a row moved to another place, a row rotated by
half, two interleaved halves, a local band first and strided columns after it.  A run that lies past the end of a CTA's part of the columns must not hide what stands behind
it.  Against the fp64 oracle."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from gpu_util import captured_kernels, dev, spmm_oracle, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu
K, N = 3072, 72


def moved_blocks(m_vec, V, seed):
    """Rows of distinct columns; every fourth one ascends."""
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(m_vec):
        c = np.sort(rng.choice(K, int(rng.integers(300, 1600)), replace=False))
        kind = i % 8
        if kind in (1, 5):     # two to five blocks in another order, most of them longer than the 64 entries that a group of lanes looks at
            cuts = np.sort(rng.choice(np.arange(1, len(c)), int(rng.integers(1, 5)), replace=False))
            blocks = np.split(c, cuts)
            c = np.concatenate([blocks[j] for j in rng.permutation(len(blocks))])
        elif kind == 2:
            c = np.roll(c, len(c) // 2)
        elif kind == 3:
            c = np.concatenate([c[::2], c[1::2]])
        elif kind == 6:        # a local band, then columns with a stride all over the row
            at = int(rng.integers(0, K - 300))
            c = np.concatenate([np.arange(at, at + 300), np.setdiff1d(np.arange(int(rng.integers(0, 9)), K, 9), np.arange(at, at + 300))])
        elif kind == 7:        # one run moved over the end of a part: 0 .. 99, 2000 .. 2200, 100 .. 1499, 2300 .. 2999
            c = np.concatenate([np.arange(100), np.arange(2000, 2201), np.arange(100, 1500), np.arange(2300, 3000)])
        rows.append(c)
    ro = np.concatenate([[0], np.cumsum([len(c) for c in rows])]).astype(np.int32)
    return cvse.CVSE(m_vec, K, V, ro, np.concatenate(rows).astype(np.int32), cvse.row_swizzle(ro, True))


@pytest.mark.parametrize("split", [None, 2, 4, 8])
@pytest.mark.parametrize("V", [1, 2, 4, 8])
def test_no_entry_is_lost(monkeypatch, V, split):
    if split:
        monkeypatch.setenv("VSPARSE_B200_SPMM", "direct")
        monkeypatch.setenv("VSPARSE_B200_SPMM_SPLIT", str(split))
    else:   # by default
        monkeypatch.delenv("VSPARSE_B200_SPMM", raising=False)
        monkeypatch.delenv("VSPARSE_B200_SPMM_SPLIT", raising=False)
    a, batch = moved_blocks(40, V, 10 * V + (split or 0)), 2
    rng = np.random.default_rng(V)
    # sums of up to 0.05 sqrt(2401) x 6 = 15: rounding them to fp16 takes 2^-8 at most, the bound on the largest difference is 0.02
    row = (a.nnz_vec * V + 7) // 8 * 8
    vals, n_cols = (0.05 * rng.standard_normal((batch, row))).astype(np.float16), N
    st = structure(a)
    for path, dtype in ((VS_PATH_CUDA_CORE, torch.float16),) + (((VS_PATH_TENSOR, torch.float32),) if V > 1 else ()):
        n_cols = 64 if path == VS_PATH_TENSOR else N
        B = rng.standard_normal((batch, K, n_cols)).astype(np.float16)
        out = torch.full((batch, a.m, n_cols), float("nan"), dtype=dtype, device="cuda:0")
        operands = dev(vals), dev(B), out
        names = captured_kernels(lambda: ops.spmm_batched(path, a.m_vec, V, n_cols, K, *st, *operands))
        assert ops.device_status() == 0 and "spmm_direct_kernel" in names and "Lb1E" in names, names
        for b in range(batch):
            assert_close(out[b].float().cpu().numpy(), spmm_oracle(a, n_cols, vals[b, :a.nnz_vec * V], B[b]), f"path {path}, entry {b}")
