"""Shards that would take another kernel than the whole call has, alone, and with it other bits: through shard.py, or inside shard.part_of, they have those of
the whole."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, dev, problem, structure
from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, cvse, ops, shard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,s", [(1, 0.8), (4, 0.7)])
@pytest.mark.parametrize("G", [2, 8])
def test_column_shards_of_dense_fp32_products(V, s, G):
    """The whole is multiplied on the tensor cores, shards of 128 columns alone would not be."""
    N, K = 1024, 4096
    a = problem(cvse.GEN_UNIFORM, 60 + V, 4096 // V, K, V, s)
    st = structure(a)
    vals = dev(cvse.fill_random((a.nnz_vec * V,), np.float32, cvse.DIST_UNIFORM, 1))
    B = torch.from_numpy(cvse.fill_random((K, N), np.float32, cvse.DIST_UNIFORM, 2, 1.0)).to(DEV)
    full = torch.empty((a.m, N), dtype=torch.float32, device=DEV)
    ops.spmm.cudaSpmm(a.m_vec, V, N, K, *st, vals, B, full)
    parts, alone = [], []
    for rank in range(G):
        B_local = shard.take_columns(B, rank, G)
        for run, to in ((lambda *x: shard.spmm_column_sharded(ops.spmm.cudaSpmm, a.m_vec, V, N, K, st, vals, *x), parts),
                        (lambda b, o: ops.spmm.cudaSpmm(a.m_vec, V, b.shape[1], K, *st, vals, b, o), alone)):
            out_local = torch.full((a.m, B_local.shape[1]), float("nan"), dtype=torch.float32, device=DEV)
            run(B_local, out_local)
            to.append(out_local)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(torch.cat(parts, dim=1), full)
    if G == 8:
        assert not torch.equal(torch.cat(alone, dim=1), full), "shards alone take the same kernel: nothing is tested"


@pytest.mark.parametrize("G", [4])
def test_batch_shards_of_dense_fp32_products(G):
    V, N, K, batch = 2, 512, 512, 8
    a = problem(cvse.GEN_UNIFORM, 5, 1024 // V, K, V, 0.6)
    st = structure(a)
    row = (a.nnz_vec * V + 7) // 8 * 8
    vals = dev(cvse.fill_random((batch, row), np.float32, cvse.DIST_UNIFORM, 1))
    B = dev(cvse.fill_random((batch, K, N), np.float32, cvse.DIST_UNIFORM, 2, 1.0))
    full, parts = (torch.full((batch, a.m, N), float("nan"), device=DEV) for _ in range(2))
    ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, V, N, K, *st, vals, B, full)
    with shard.part_of(batch=batch):
        for b0, cnt in shard.batch_shards(batch, G):
            ops.spmm_batched(VS_PATH_CUDA_CORE, a.m_vec, V, N, K, *st, vals[b0:b0 + cnt].contiguous(), B[b0:b0 + cnt].contiguous(), parts[b0:b0 + cnt])
    torch.cuda.synchronize()
    assert torch.equal(parts, full)


@pytest.mark.parametrize("G", [2, 8])
def test_batch_shards_of_attention(G):
    """128 heads fill the GPU with one warp to a vector-row; 16 of them alone take four."""
    V, d, n, heads = 8, 64, 1024, 128
    a = problem(cvse.GEN_BAND, 8, n // V, n, V, 0.9, band=128)
    st = structure(a)
    q, k, v = (torch.from_numpy(cvse.fill_random((heads, n, d), np.float16, cvse.DIST_NORMAL, 20 + i, 1.0)).to(DEV) for i in range(3))
    ws = torch.empty((heads, a.nnz_vec * V), dtype=torch.float16, device=DEV)

    def run(h0, cnt):
        o = torch.full((cnt, n, d), float("nan"), dtype=torch.float16, device=DEV)
        ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *st, *(x[h0:h0 + cnt].contiguous() for x in (q, k, v)), o, ws[:cnt], 0.125)
        return o

    full = run(0, heads)
    with shard.part_of(batch=heads):
        parts = [run(h0, cnt) for h0, cnt in shard.batch_shards(heads, G)]
    alone = [run(h0, cnt) for h0, cnt in shard.batch_shards(heads, G)]
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(torch.cat(parts), full)
    if G == 8:
        assert not torch.equal(torch.cat(alone), full), "shards alone take the same number of warps: nothing is tested"
