"""Softmax of large scores in fixed-mask attention: probabilities as near to those of the same fp16 scores in 64 bits as their own roundings to fp16
allow, however large the scores (the sum of a row's exponentials, next to scores of thousands, must not be blurred)."""
import numpy as np
import pytest
import torch

from gpu_util import DEV, custom, dev, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", ["1", "2", "4"])
@pytest.mark.parametrize("scale", [1.0, 0.125, 0.0009, -1.0, 0.0])   # scores times scale around 57000, 7000, 50; the last two operator by operator
@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("d", [64, 128])
def test_probabilities(monkeypatch, d, warps, scale, backward):
    """Queries and keys with one element each, so that the fp16 scores are known exactly: neighbouring fp16 numbers around 57000, of which several share
    a row's maximum."""
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "fused")
    monkeypatch.setenv("VSPARSE_B200_ATTENTION_WARPS", warps)
    V, n = 8, 512
    a = custom([3, 17, 0, 40, 100, 200, 300, 31, 1], n, V, seed=4)
    rng = np.random.default_rng(1)
    q, k, v, go = np.zeros((a.m, d), np.float16), np.zeros((n, d), np.float16), rng.standard_normal((n, d)).astype(np.float16), np.zeros((a.m, d), np.float16)
    q[:, 0] = 1.0 + rng.integers(0, 8, a.m) / 64
    k[:, 0] = np.sign(scale or 1.0) * (55000 - 32 * rng.integers(0, 3, n))
    go[:, 5] = rng.standard_normal(a.m)
    st, size = structure(a), a.nnz_vec * V
    probs, grads = (torch.full((size,), float("nan"), dtype=torch.float16, device=DEV) for _ in range(2))
    out, gv, gk = (torch.full((x, d), float("nan"), dtype=torch.float16, device=DEV) for x in (a.m, n, n))
    if backward:
        ops.attention_cvse_backward(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *st, *(dev(x) for x in cvse.transpose(a)), dev(q), dev(k), dev(v), dev(go), out,
                                    gk, gv, probs, grads, scale)
    else:
        ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, n, d, a.nnz_vec, *st, dev(q), dev(k), dev(v), out, probs, scale)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    got = probs.cpu().numpy().astype(np.float64).reshape(-1, V)
    # a rounding to fp16 is 2^-11 of the value (2^-25 among its subnormals): one in one kernel, of the exponential, of 1 / sum and of their product
    # operator by operator; exponents and sums of up to 300 terms in fp32: 2^-16
    roundings = 1 if scale > 0 else 3
    for i in range(a.m_vec):
        cols, at = a.col_indices[a.row_offsets[i]:a.row_offsets[i + 1]], slice(a.row_offsets[i], a.row_offsets[i + 1])
        if len(cols) == 0:
            assert bool((out[i * V:(i + 1) * V] == 0).all())
            continue
        rows = slice(i * V, (i + 1) * V)
        s = np.outer(k[cols, 0].astype(np.float64), q[rows, 0].astype(np.float64)).astype(np.float16).astype(np.float64) * np.float64(np.float32(scale))
        e = np.exp(s - s.max(axis=0))
        p = e / e.sum(axis=0)
        assert np.all(np.abs(got[at] - p) <= p * (roundings * 2.0 ** -11 + 2.0 ** -16) + 2.0 ** -23), i
        if not backward:   # weights of a relative error that is the same for all keys at most; the result is rounded too
            want = p.T @ v[cols].astype(np.float64)
            bound = p.T @ np.abs(v[cols].astype(np.float64)) * (roundings * 2.0 ** -11 + 2.0 ** -15) + np.abs(want) * 2.0 ** -11 + 2.0 ** -20
            assert np.all(np.abs(out[rows].cpu().numpy().astype(np.float64) - want) <= bound), i
