"""Attention's backward where results share memory with one another (a buffer for what is not wanted): they are written one after the other, by the operators dV, dQ, dK,
by the one kernel and the products behind it dQ, dV, dK, and the last one stands."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, custom, dev, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["steps", "fused"])
@pytest.mark.parametrize("heads,n,d", [(3, 264, 64), (20, 520, 128)])
def test_the_last_one_stands(monkeypatch, form, heads, n, d):
    monkeypatch.setenv("VSPARSE_B200_SPMM_T", "dense")
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", form)
    V = 4
    a = custom([4 * (7 * i % (n // 16)) for i in range(n // V)], n, V, seed=n + V)
    q, k, v, go = (dev(cvse.fill_random((heads, n, d), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0)) for i in range(4))
    s, t = structure(a), [dev(x) for x in cvse.transpose(a)]

    def run(same):
        p, g = (torch.zeros(heads, a.nnz_vec * V, dtype=torch.float16, device=DEV) for _ in range(2))
        grads = {x: torch.full((heads, n, d), float("nan"), dtype=torch.float16, device=DEV) for x in "qkv"}
        for x in same[1:]:
            grads[x] = grads[same[0]]
        ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *s, *t, q, k, v, go, grads["q"], grads["k"], grads["v"], p, g, 0.125)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        return grads

    want = run("")
    for same in ("kv", "qv", "qk", "qkv"):
        got = run(same)
        for x in set("qkv") - set(same) | {"k" if "k" in same else "q" if form == "steps" else "v"}:
            assert torch.equal(got[x], want[x]), (same, x)
