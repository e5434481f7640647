"""A pipeline wait of the FP64-accurate product that gives up
(IPT_GB300_SPIN_LIMIT=1: after a single poll; the kernel sets its error flag,
drains its own copies and returns) ends a plain, ACX or FP64 block solve with
the CUDA-error status, never with success and a NaN block; the next call on
the same context succeeds."""
import ctypes as C

import pytest

from block_ipt_gb300 import _lib, api, workloads

import numpy as np

pytestmark = pytest.mark.gpu

N, K = 2048, 16


def fixed(lib, dH, handle):
    vec, val = C.c_void_p(), C.c_void_p()
    st = lib.ipt_cuda_device(dH, N, K, 3, handle, C.byref(vec), C.byref(val))
    lib.ipt_cuda_free_device_result(vec, val)
    return st


def tolerance(lib, dH, handle):
    vec, val = C.c_void_p(), C.c_void_p()
    it, res = C.c_int(0), C.c_double(0.0)
    st = lib.ipt_cuda_device_tol(dH, N, K, 1e-12, 200, handle, C.byref(vec), C.byref(val),
                                 C.byref(it), C.byref(res))
    lib.ipt_cuda_free_device_result(vec, val)
    return st


def acx(lib, dH, handle):
    res = _lib.ACXCudaResult()
    lib.acx_cuda_reset_result(C.byref(res))
    st = lib.acx_cuda_device_tol(dH, N, K, 1e-12, 200, handle, C.byref(res))
    lib.acx_cuda_free_result(C.byref(res))
    return st


def block(lib, dH, handle):
    import torch
    X = torch.empty(K, N, dtype=torch.float64, device="cuda")
    w = torch.empty(K, dtype=torch.float64, device="cuda")
    try:
        api.block_solve_dense_device(dH.value, N, K, X.data_ptr(), w.data_ptr(), "fp64")
    except _lib.IPTError as exc:
        return exc.status
    return 0


@pytest.mark.parametrize("entry", [fixed, tolerance, acx, block], ids=lambda f: f.__name__)
def test_wait_limit_gives_error_status(cuda, monkeypatch, entry):
    torch = cuda
    H, _ = workloads.dense_config0(N, seed=5)
    t = torch.from_numpy(np.asfortranarray(H).T.copy()).cuda()
    dH, handle = C.c_void_p(t.data_ptr()), C.c_void_p(torch.cuda.current_blas_handle())
    lib = _lib.load()
    monkeypatch.setenv("IPT_GB300_SPIN_LIMIT", "1")
    # 3: CUDA error, in both headers
    assert entry(lib, dH, handle) == 3
    monkeypatch.delenv("IPT_GB300_SPIN_LIMIT")
    torch.cuda.synchronize()
    assert entry(lib, dH, handle) == 0
