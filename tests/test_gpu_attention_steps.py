"""Fixed-mask attention operator by operator on the tensor path, forward and backward, against the fp64 oracle, and the calls that go there by
themselves: other head dimensions, operands on 16-byte boundaries, dense masks of short vectors, the choice of the caller."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close
from gpu_util import DEV, captured_kernels, dev, problem, structure
from vectorsparse_b200 import VS_PATH_TENSOR, cvse, ops

pytestmark = pytest.mark.gpu


class Layer:
    def __init__(self, V, d, n, heads, seed=6):
        self.V, self.d, self.n, self.heads = V, d, n, heads
        self.a = a = problem(cvse.GEN_BAND, seed, n // V, n, V, 0.8, band=64)
        assert a.nnz_vec * V % 8 == 0
        self.host = [cvse.fill_random((heads, n, d), np.float16, cvse.DIST_NORMAL, 10 + i, 1.0) for i in range(4)]
        self.q, self.k, self.v, self.go = (dev(x) for x in self.host)
        self.st, self.t = structure(a), [dev(x) for x in cvse.transpose(a)]
        self.scale = d ** -0.5
        self.out, self.gq, self.gk, self.gv = (torch.full((heads, n, d), float("nan"), dtype=torch.float16, device=DEV) for _ in range(4))
        self.ws_p, self.ws_g = (torch.empty((heads, a.nnz_vec * V), dtype=torch.float16, device=DEV) for _ in range(2))

    def forward(self):
        ops.attention_cvse(VS_PATH_TENSOR, self.a.m_vec, self.V, self.n, self.d, self.a.nnz_vec, *self.st, self.q, self.k, self.v, self.out, self.ws_p, self.scale)

    def backward(self):
        ops.attention_cvse_backward(VS_PATH_TENSOR, self.a.m_vec, self.V, self.n, self.d, self.a.nnz_vec, *self.st, *self.t, self.q, self.k, self.v,
                                    self.go, self.gq, self.gk, self.gv, self.ws_p, self.ws_g, self.scale)

    def check(self, heads):
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        a = self.a
        for h in heads:
            q, k, v, go = (x[h].astype(np.float32) for x in self.host)
            want = [oracle.attention(a.m_vec, self.V, self.d, self.d, a.row_offsets, a.col_indices, q, k, v, self.scale),
                    *oracle.attention_backward(a.m_vec, self.V, self.d, a.row_offsets, a.col_indices, q, k, v, go, self.scale)]
            for got, w, what in zip((self.out, self.gq, self.gk, self.gv), want, ("out", "dQ", "dK", "dV")):
                assert_close(got[h].float().cpu().numpy(), w, f"{what}, head {h}")

    def fused(self):
        return ["attention_kernel" in captured_kernels(f) for f in (self.forward, self.backward)]


@pytest.mark.parametrize("V", [2, 4, 8])
@pytest.mark.parametrize("d", [64, 128])
def test_by_choice_of_the_caller(monkeypatch, V, d):
    layer = Layer(V, d, 512, 2)
    assert layer.fused() == [True, True]
    monkeypatch.setenv("VSPARSE_B200_ATTENTION", "steps")
    assert layer.fused() == [False, False]
    layer.forward()
    layer.backward()
    layer.check(range(2))


def test_other_head_dimensions():
    layer = Layer(8, 192, 512, 2)
    assert layer.fused() == [False, False]
    layer.check(range(2))


def test_operands_on_16_byte_boundaries():
    layer = Layer(8, 64, 512, 2)
    buf = torch.empty(layer.k.numel() + 8, dtype=torch.float16, device=DEV)
    buf[8:] = layer.k.view(-1)
    layer.k = buf[8:].view(layer.k.shape)
    assert layer.fused() == [False, False]
    layer.check(range(2))


@pytest.mark.parametrize("V,d,heads,fused", [(4, 128, 28, True), (4, 128, 30, False), (2, 64, 28, True), (2, 64, 30, False), (4, 64, 60, False), (8, 64, 128, True), (8, 128, 64, False)])
def test_dense_masks(V, d, heads, fused):
    """20 % of 1024 keys, on both sides of three million of them (twice as many at d = 128)."""
    layer = Layer(V, d, 1024, heads)
    assert layer.fused() == [fused, fused]
    if V < 8:
        layer.check((0, heads - 1))


def test_sparse_masks_stay_one_kernel():
    layer = Layer(2, 64, 1024, 80)
    layer.a = problem(cvse.GEN_BAND, 6, 512, 1024, 2, 0.89, band=64)
    layer.st, layer.t = structure(layer.a), [dev(x) for x in cvse.transpose(layer.a)]
    assert layer.a.nnz_vec * 80 > 3000000 and layer.fused() == [True, True]
