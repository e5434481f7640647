"""FP64 FMAs on request (IPT_GB300_FP64_DFMA=1 or
IPT_GB300_ACCURATE_PRODUCT=fp64) in the plain, ACX and block-solver FP64
solves: every entry of the vectors to FP64's own relative accuracy on a graded
matrix, and no digit words laid out.

Tolerance: an FP64 sum of n terms is off by at most n 2^-53 of the sum of
their magnitudes; with the diagonal carried through and taken off again that
sum is at most 4 |X_ic| / |g_ic| on this matrix (couplings 5e-4), and a
contracting map adds at most as much again: 16 n 2^-53 covers a fixed point.
"""
import ctypes as C

import numpy as np
import pytest

from block_ipt_gb300 import _lib, api
from tests.conftest import _load_cudart, device_to_host

pytestmark = pytest.mark.gpu

KNOBS = [("IPT_GB300_FP64_DFMA", "1"), ("IPT_GB300_ACCURATE_PRODUCT", "fp64")]


def graded(n, decades, seed):
    """Diagonal from 1 to 10^decades, couplings 5e-4 sqrt(d_i d_j) N(0, 1)."""
    rng = np.random.default_rng(seed)
    d = np.logspace(0, decades, n)
    A = np.triu(rng.standard_normal((n, n)), 1)
    H = (A + A.T) * 5e-4 * np.sqrt(d)[:, None] * np.sqrt(d)[None, :]
    H[np.arange(n), np.arange(n)] = d
    return H


def fixed_point(H, k, steps, X=None):
    L = H.astype(np.longdouble)
    n = H.shape[0]
    d = np.diag(L).copy()
    D = L - np.diag(d)
    X = np.eye(n, k, dtype=np.longdouble) if X is None else X
    gap = d[None, :k] - d[:, None]
    gap[np.arange(k), np.arange(k)] = 1
    for _ in range(steps):
        Y = D @ X
        X = (Y - X * np.diagonal(Y[:k])[None, :]) / gap
        X[np.arange(k), np.arange(k)] = 1
    return X


def plain(torch, H, k, iterations):
    lib = _lib.load()
    n = H.shape[0]
    dH = torch.from_numpy(np.asfortranarray(H).T.copy()).cuda()
    vec, val = C.c_void_p(), C.c_void_p()
    st = lib.ipt_cuda_device(C.c_void_p(dH.data_ptr()), n, k, iterations,
                             C.c_void_p(torch.cuda.current_blas_handle()), C.byref(vec),
                             C.byref(val))
    assert st == 0, _lib.status_string(st)
    torch.cuda.synchronize()
    X = device_to_host(vec, np.zeros((n, k), order="F"))
    lib.ipt_cuda_free_device_result(vec, val)
    return X


def acx(torch, H, k):
    lib = _lib.load()
    n = H.shape[0]
    dH = torch.from_numpy(np.asfortranarray(H).T.copy()).cuda()
    res = _lib.ACXCudaResult()
    lib.acx_cuda_reset_result(C.byref(res))
    st = lib.acx_cuda_device_tol(C.c_void_p(dH.data_ptr()), n, k, 1e-15, 30,
                                 C.c_void_p(torch.cuda.current_blas_handle()), C.byref(res))
    assert st == 0, _lib.status_string(st)
    X = device_to_host(C.c_void_p(res.d_vectors), np.zeros((n, k), order="F"))
    lib.acx_cuda_free_result(C.byref(res))
    return X


@pytest.mark.parametrize("knob", KNOBS)
@pytest.mark.parametrize("decades", [12, 20])
def test_entries_on_a_graded_matrix(cuda, monkeypatch, knob, decades):
    monkeypatch.setenv(*knob)
    n, k = 300, 8
    H = graded(n, decades, 1)
    for steps in (1, 12):
        X = plain(cuda, H, k, steps)
        Xr = fixed_point(H, k, steps)
        rel = np.abs(X - Xr) / np.maximum(np.abs(Xr), np.longdouble(1e-300))
        assert rel.max() <= 16 * n * 2.0 ** -53
    Xr = fixed_point(H, k, 40)
    rel = np.abs(acx(cuda, H, k) - Xr) / np.abs(Xr)
    assert rel.max() <= 16 * n * 2.0 ** -53


def pool_peak(torch, call):
    """Largest use of the library's stream-ordered pool during `call`, bytes."""
    rt = _load_cudart()
    pool = C.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    torch.cuda.synchronize()
    value = C.c_ulonglong(0)
    used_high = 8  # cudaMemPoolAttrUsedMemHigh
    assert rt.cudaMemPoolSetAttribute(pool, used_high, C.byref(value)) == 0
    call()
    torch.cuda.synchronize()
    assert rt.cudaMemPoolGetAttribute(pool, used_high, C.byref(value)) == 0
    return value.value


def block_case(torch, n, k):
    rng = np.random.default_rng(2)
    A = rng.standard_normal((n, n)) * (0.05 / np.sqrt(n))
    H = A + A.T + np.diag(np.arange(1.0, n + 1))
    dH = torch.from_numpy(H).cuda()
    X = torch.empty(k, n, dtype=torch.float64, device="cuda")
    w = torch.empty(k, dtype=torch.float64, device="cuda")

    def solve():
        api.block_solve_dense_device(dH.data_ptr(), n, k, X.data_ptr(), w.data_ptr(), "fp64")

    return H, solve, w


def test_block_solver_lays_the_digits_out_once(cuda):
    """8 n^2 bytes of digit words, and less than half of that for the rest."""
    n, k = 4096, 8
    H, solve, w = block_case(cuda, n, k)
    peak = pool_peak(cuda, solve)
    assert 8 * n * n <= peak < 12 * n * n
    assert np.abs(w.cpu().numpy() - np.linalg.eigvalsh(H)[:k]).max() <= 1e-10 * np.abs(H).sum(1).max()


@pytest.mark.parametrize("knob", KNOBS)
def test_block_solver_lays_out_no_digits(cuda, monkeypatch, knob):
    monkeypatch.setenv(*knob)
    n, k = 2048, 8
    H, solve, w = block_case(cuda, n, k)
    assert pool_peak(cuda, solve) < 8 * n * n
    # eigenvalues to the solver's residual tolerance
    assert np.abs(w.cpu().numpy() - np.linalg.eigvalsh(H)[:k]).max() <= 1e-10 * np.abs(H).sum(1).max()
