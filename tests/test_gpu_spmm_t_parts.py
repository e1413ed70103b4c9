"""Transposed products that are small by themselves but parts of one that is not: inside shard.part_of, and one after the other in attention's backward by its operators,
they are multiplied as the whole is, with its bits."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, captured_kernels, custom, dev, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops, shard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("by", ["columns", "batch"])
def test_parts_below_the_line(monkeypatch, V, by):
    """512 x 512 x 1024 (or 4 x 256) is past 1e8 multiply-adds, a quarter of it is not."""
    monkeypatch.delenv("VSPARSE_B200_SPMM_T", raising=False)
    m, n, N, batch = 512, 512, 1024 if by == "columns" else 256, 1 if by == "columns" else 4
    a = custom([n // 3] * (m // V), n, V, seed=V)
    t = [dev(x) for x in cvse.transpose(a)]
    vals = dev(cvse.fill_random((batch, a.nnz_vec * V), np.float16, cvse.DIST_NORMAL, 3, 1.0))
    rhs = dev(cvse.fill_random((batch, a.m, N), np.float16, cvse.DIST_NORMAL, 4, 1.0))
    full, parts, alone = (torch.full((batch, n, N), float("nan"), device=DEV) for _ in range(3))
    ops.spmm_t(a.m_vec, V, N, n, *t, vals, rhs, full)

    def in_parts(to):
        if by == "batch":
            for b in range(batch):
                ops.spmm_t(a.m_vec, V, N, n, *t, vals[b:b + 1], rhs[b:b + 1], to[b:b + 1])
        else:
            for c in range(0, N, 256):
                out = torch.empty((1, n, 256), device=DEV)
                ops.spmm_t(a.m_vec, V, 256, n, *t, vals, rhs[..., c:c + 256].contiguous(), out)
                to[..., c:c + 256] = out
    in_parts(alone)
    with shard.part_of(**{by: N if by == "columns" else batch}):
        in_parts(parts)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(parts, full)
    if m // V <= 512 and V >= 4:
        assert not torch.equal(alone, full), "parts alone take the same kernel: nothing is tested"


def test_backward_by_the_operators(monkeypatch):
    """dQ or dK over dO or P: the two transposed products one after the other, each small, with the bits of both at once."""
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "steps")
    monkeypatch.delenv("VSPARSE_B200_SPMM_T", raising=False)
    V, heads, n, d = 4, 2, 264, 64
    a = custom([4 * (7 * i % (n // 16)) for i in range(n // V)], n, V, seed=n + V)
    q, k, v, go = (dev(cvse.fill_random((heads, n, d), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0)) for i in range(4))
    s, t = structure(a), [dev(x) for x in cvse.transpose(a)]

    def run(over):
        grad_out = go.clone()
        ws_p, ws_g = (torch.zeros(heads * max(a.nnz_vec * V, n * d), dtype=torch.float16, device=DEV) for _ in range(2))
        p, g = (w[:heads * a.nnz_vec * V].view(heads, -1) for w in (ws_p, ws_g))
        gq, gk, gv = (torch.full((heads, n, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(3))
        if over == "q on grad_out":
            gq = grad_out
        if over == "k on p":
            gk = ws_p[:heads * n * d].view(heads, n, d)
        names = captured_kernels(lambda: ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *s, *t, q, k, v, grad_out, gq, gk, gv, p, g, 0.125))
        assert ops.device_status() == 0
        return names.count("dense_plan_kernelILb1E"), [x.clone() for x in (gq, gk, gv)]

    plans, want = run("")
    assert plans == 1
    for over in ("q on grad_out", "k on p"):
        plans, got = run(over)
        assert plans == 2
        assert all(torch.equal(x, w) for x, w in zip(got, want)), over
