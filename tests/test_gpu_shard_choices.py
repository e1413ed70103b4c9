"""fp16 products whose shards, by their own sizes, would take another kernel, or share tiles among another number of CTAs, than the whole: inside shard.part_of they have its
bits.  fp32 results show every difference in the order of the sums."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, dev, problem, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops, shard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,V,K,N,s,G", [(1180, 2, 1966, 640, 0.8, 2), (656, 2, 1460, 1344, 0.78, 4), (908, 2, 1511, 896, 0.57, 2), (640, 2, 2048, 1024, 0.8, 4),
                                         (640, 4, 2048, 1024, 0.8, 4), (256, 8, 4095, 512, 0.7, 8)])
def test_column_shards(m, V, K, N, s, G):
    """A whole whose matrix is laid out first and shards that the one-kernel form would take, with shared tiles; and the reverse: shared by fewer CTAs than a shard alone."""
    a = problem(cvse.GEN_UNIFORM, m + N, m // V, K, V, s)
    st = structure(a)
    vals = dev(cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.5))
    B = dev(cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 1.0))
    full = torch.empty((a.m, N), dtype=torch.float32, device=DEV)
    ops.spmm.wmmaSpmm(a.m_vec, V, N, K, *st, vals, B, full)
    parts = []
    for rank in range(G):
        B_local = shard.take_columns(B, rank, G)
        out_local = torch.full((a.m, B_local.shape[1]), float("nan"), dtype=torch.float32, device=DEV)
        shard.spmm_column_sharded(ops.spmm.wmmaSpmm, a.m_vec, V, N, K, st, vals, B_local, out_local)
        parts.append(out_local)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(torch.cat(parts, dim=1), full)


@pytest.mark.parametrize("V", [1, 2])
def test_column_shards_behind_the_cuda_core_entry_point(V):
    """Its choice by density knows the whole's tiles as well."""
    m, K, N, G = 640, 2048, 1024, 8
    a = problem(cvse.GEN_UNIFORM, V, m // V, K, V, 0.8)
    st = structure(a)
    vals = dev(cvse.fill_random((a.nnz_vec * V,), np.float16, cvse.DIST_NORMAL, 1, 0.5))
    B = dev(cvse.fill_random((K, N), np.float16, cvse.DIST_NORMAL, 2, 1.0))
    full = torch.empty((a.m, N), dtype=torch.float16, device=DEV)
    ops.spmm.cudaSpmm(a.m_vec, V, N, K, *st, vals, B, full)
    parts = []
    for rank in range(G):
        B_local = shard.take_columns(B, rank, G)
        out_local = torch.full((a.m, B_local.shape[1]), float("nan"), dtype=torch.float16, device=DEV)
        shard.spmm_column_sharded(ops.spmm.cudaSpmm, a.m_vec, V, N, K, st, vals, B_local, out_local)
        parts.append(out_local)
    assert torch.equal(torch.cat(parts, dim=1), full)


@pytest.mark.parametrize("m,V,K,N,batch", [(512, 2, 1536, 512, 2), (256, 4, 2048, 128, 40), (128, 8, 1000, 64, 4)])
def test_batch_shards(m, V, K, N, batch):
    a = problem(cvse.GEN_UNIFORM, m + N, m // V, K, V, 0.8)
    st = structure(a)
    row = (a.nnz_vec * V + 7) // 8 * 8
    vals = dev(cvse.fill_random((batch, row), np.float16, cvse.DIST_NORMAL, 1, 0.5))
    B = dev(cvse.fill_random((batch, K, N), np.float16, cvse.DIST_NORMAL, 2, 1.0))
    full, parts = (torch.full((batch, a.m, N), float("nan"), device=DEV) for _ in range(2))
    ops.spmm_batched(VS_PATH_TENSOR, a.m_vec, V, N, K, *st, vals, B, full)
    with shard.part_of(batch=batch):
        for b0, cnt in shard.batch_shards(batch, 2) + [(0, 1), (batch - 1, 1)]:
            ops.spmm_batched(VS_PATH_TENSOR, a.m_vec, V, N, K, *st, vals[b0:b0 + cnt], B[b0:b0 + cnt], parts[b0:b0 + cnt])
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(parts, full)
