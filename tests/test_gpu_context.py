"""Which CUDA context the library works in: the caller's current one, and the device's primary one for a thread that has none."""
import ctypes
import threading

import pytest
import torch

from gpu_util import DEV
from vectorsparse_b200 import _lib

pytestmark = pytest.mark.gpu


def in_thread(f):
    """f() on a thread that has made no CUDA call yet."""
    result = []
    t = threading.Thread(target=lambda: result.append(f()))
    t.start()
    t.join()
    return result[0]


def test_a_call_leaves_the_callers_context_current():
    torch.zeros(1, device=DEV)
    lib, cu = _lib.lib(), ctypes.CDLL("libcuda.so.1")
    assert lib.vs_release_scratch(None, 0) == 0   # the device's figures are read in its primary context

    def call():
        own, current = ctypes.c_void_p(), ctypes.c_void_p()
        assert cu.cuCtxCreate_v2(ctypes.byref(own), 0, 0) == 0
        try:
            rc = lib.vs_release_scratch(None, 0)
            assert cu.cuCtxGetCurrent(ctypes.byref(current)) == 0
        finally:
            assert cu.cuCtxDestroy_v2(own) == 0
        return rc, own.value == current.value

    assert in_thread(call) == (0, True)


def test_a_thread_without_a_context_gets_one():
    lib, cu = _lib.lib(), ctypes.CDLL("libcuda.so.1")
    torch.zeros(1, device=DEV)

    def call():
        current = ctypes.c_void_p()
        rc = lib.vs_release_scratch(None, 0)
        assert cu.cuCtxGetCurrent(ctypes.byref(current)) == 0
        return rc, current.value is not None

    assert in_thread(call) == (0, True)
