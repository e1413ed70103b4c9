"""The plan of the dense SDDMM, the mask as words of 32 columns: rows planned by a warp and by a CTA, whose last word is partly empty, in ascending order, in
another, with columns named twice; V = 1 to 8, both entry points, against the fp64 oracle."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, captured_kernels, custom, dev, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("n,lens,share", [(33, [0, 1, 31, 32, 33, 5], 1), (320, [1, 200, 0, 64, 33, 190], 1), (320, [320, 257, 0, 310, 319, 2], 8),
                                          (1000, [1000, 999, 0, 129, 1, 500], 8), (8192, [8192, 0, 300], 8), (8161, [8000, 1, 33], 8)])
def test_words(monkeypatch, V, n, lens, share):
    monkeypatch.setenv("VSPARSE_B200_SDDMM", "dense")
    a, k, batch = custom(np.resize(lens, 71 if n < 2000 else 5), n, V, seed=V), 64, 2
    rng = np.random.default_rng(n)
    for i, order in ((1, rng.permutation), (3, lambda c: np.sort(rng.choice(c, c.size))), (4, lambda c: rng.choice(c, c.size))):   # disorder, twins in order, both
        if i < a.m_vec:
            row = slice(a.row_offsets[i], a.row_offsets[i + 1])
            if row.stop > row.start:
                a.col_indices[row] = order(a.col_indices[row])
    lhs, rhs = (rng.standard_normal((batch, rows, k)).astype(np.float16) for rows in (a.m, n))
    st, size = structure(a), (a.nnz_vec * V + 7) // 8 * 8
    for path, dtype in ((VS_PATH_CUDA_CORE, torch.float16),) if V == 1 else ((VS_PATH_CUDA_CORE, torch.float16), (VS_PATH_TENSOR, torch.float32)):
        out = torch.full((batch * size + 64,), float("nan"), dtype=dtype, device=DEV)
        operands = dev(lhs), dev(rhs), out[:batch * size].view(batch, size)
        names = captured_kernels(lambda: ops.sddmm_batched(path, a.m_vec, k, n, a.nnz_vec, *st, *operands, V))
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        assert f"sddmm_cell_plan_kernelILi{share}E" in names and "sddmm_pair_kernel" in names
        assert bool(torch.isnan(out[batch * size:]).all())
        for b in range(batch):
            want = oracle.sddmm(a.m_vec, k, V, a.row_offsets, a.col_indices, lhs[b].astype(np.float32), rhs[b].astype(np.float32), acc="f64")
            assert_close(out[b * size:b * size + a.nnz_vec * V].float().cpu().numpy(), want, f"entry {b}")
