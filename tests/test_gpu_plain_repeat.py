"""The tensor-core product of the plain FP64 path gives the same bits in every
run: its partial sums are added in a fixed order, and no stage of its pipeline
may overtake another (k_oz.cu)."""
import ctypes as C

import pytest

from block_ipt_gb300 import _lib
from tests.conftest import device_to_host

import numpy as np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1501, 64), (4096, 16), (2000, 130)])
def test_same_bits_in_every_run(cuda, n, k):
    torch = cuda
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    A = torch.triu(torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64), 1)
    H = 0.02 * (A + A.T) * torch.exp(-(i[:, None] - i[None, :]).abs() / 256)
    H.diagonal().copy_(i)
    lib = _lib.load()
    handle = C.c_void_p(torch.cuda.current_blas_handle())
    first = None
    for _ in range(6):
        vec, val = C.c_void_p(), C.c_void_p()
        st = lib.ipt_cuda_device(C.c_void_p(H.data_ptr()), n, k, 5, handle, C.byref(vec),
                                 C.byref(val))
        assert st == 0, _lib.status_string(st)
        torch.cuda.synchronize()
        X = device_to_host(vec, np.zeros((n, k), order="F"))
        lib.ipt_cuda_free_device_result(vec, val)
        if first is None:
            first = X
        assert (X.view(np.int64) == first.view(np.int64)).all()
