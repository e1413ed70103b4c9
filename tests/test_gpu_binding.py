"""The extension between torch tensors and the library: it gives other Python threads their turn, and what it refuses is refused
with the same errors as ever."""
import ctypes
import subprocess
import threading

import pytest
import torch

from gpu_util import DEV
from vectorsparse_b200 import _binding, ops

pytestmark = pytest.mark.gpu

# stands in for vs_softmax_cvse: returns 0 once the flag is up, -77 if nobody has raised it after five seconds
WAITER = """
#include <time.h>
volatile int entered, flag;
int waiter(int a, int b, int c, const void *d, const void *e, const void *f, void *g, float h, int i, long long j, void *k) {
    struct timespec ms = {0, 1000000};
    entered = 1;
    for (int n = 0; n < 5000 && !flag; ++n) nanosleep(&ms, 0);
    return flag ? 0 : -77;
}
"""


def test_other_threads_run_while_a_call_blocks(tmp_path):
    (tmp_path / "waiter.c").write_text(WAITER)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(tmp_path / "waiter.so"), str(tmp_path / "waiter.c")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "waiter.so"))
    entered, flag = ctypes.c_int.in_dll(lib, "entered"), ctypes.c_int.in_dll(lib, "flag")
    waiter = ctypes.cast(lib.waiter, ctypes.c_void_p).value
    index, x = torch.zeros(8, dtype=torch.int32, device=DEV), torch.zeros(8, device=DEV)

    def raise_flag():
        while not entered.value:
            pass
        flag.value = 1

    thread = threading.Thread(target=raise_flag)
    _binding.bind(*[waiter] * 7)
    try:
        thread.start()
        rc = _binding.softmax(1, 8, index, index, x, x, 1.0)
    finally:
        ops._bind()
        thread.join()
    assert rc == 0


def test_what_the_binding_refuses_gets_the_operators_errors():
    """The wrong type, device, layout, size and element type, and arguments that only look like integers."""
    i, x = torch.zeros(16, dtype=torch.int32, device=DEV), torch.zeros(64, dtype=torch.float16, device=DEV)

    def spmm(m_vec=1, ri=i, ro=i, ci=i, values=x, rhs=x, out=x, nnz=1):
        return ops.spmm.wmmaSpmm(m_vec, 8, 8, 8, ri, ro, ci, values, rhs, out, nnz)

    for error, arguments in ((TypeError, dict(values=x.cpu())), (TypeError, dict(ci=i.long())),
                             (TypeError, dict(rhs=x.float())), (ValueError, dict(values=x[::2])), (ValueError, dict(ro=i[:1])),
                             (ValueError, dict(m_vec=2)), (ValueError, dict(nnz=17)), (ops._lib.VsError, dict(out=x.to(torch.int16)))):
        with pytest.raises(error):
            spmm(**arguments)
    with pytest.raises(ops._lib.VsError):   # taken by the binding, refused by the library: a dense width of 8
        spmm()
