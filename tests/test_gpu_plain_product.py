"""The plain FP64 path's tensor-core product and fused IPT update through
ipt_cuda_device, at the edges of its tiles: rows around multiples of 128 (row
tile), 32 (K stage), 256 and 1024 (update blocks), columns around 16 and 32
(column groups), general (non-symmetric) matrices, against the same map in
extended precision.

Tolerance: an entry of Delta X has an absolute error of at most
n (2^-56 2^e 2^f 2 + 2^-64 ...) + 2^-52 |y| <= n 2^-53 max|Delta| max|X|
(e, f the binades above the row's and column's largest entries), the map
scales it by |g|, and a contracting map (checked: the sums |g| |Delta| stay
below 1/2) carries an error on at most once more in full: 4 n 2^-53 max|g|
max|Delta| max|X| covers any number of steps.
"""
import ctypes as C

import numpy as np
import pytest

from block_ipt_gb300 import _lib
from tests.conftest import device_to_host

pytestmark = pytest.mark.gpu


def run(torch, H, k, iterations):
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
    v = device_to_host(val, np.zeros(k))
    lib.ipt_cuda_free_device_result(vec, val)
    return X, v


def reference(H, k, iterations):
    L = H.astype(np.longdouble)
    n = H.shape[0]
    d = np.diag(L).copy()
    D = L - np.diag(d)
    X = np.eye(n, k, dtype=np.longdouble)
    gap = d[None, :k] - d[:, None]
    gap[np.arange(k), np.arange(k)] = 1
    for _ in range(iterations):
        Y = D @ X
        X = (Y - X * np.diagonal(Y[:k])[None, :]) / gap
        X[np.arange(k), np.arange(k)] = 1
    return X.astype(np.float64), np.diagonal((L @ X)[:k]).astype(np.float64)


SHAPES = [(1, 1), (2, 2), (31, 5), (33, 16), (127, 17), (128, 32), (129, 33), (257, 1),
          (384, 48), (511, 65), (1025, 31), (1300, 9)]


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("wide", [False, True])
def test_iterates(cuda, n, k, wide):
    rng = np.random.default_rng(1000 * n + k)
    H = rng.standard_normal((n, n)) * (0.2 / n)
    if wide:  # rows over many binades
        H *= np.exp(-rng.uniform(0, 30, (n, 1)))
    d = np.arange(n) + 0.3 * rng.uniform(size=n)
    H[np.arange(n), np.arange(n)] = d
    k = min(n, k)
    gap = np.abs(d[None, :k] - d[:, None])
    gap[np.arange(k), np.arange(k)] = np.inf
    D = np.abs(H - np.diag(d))
    assert (D.sum(axis=1)[:, None] / gap).max() < 0.5 or n == 1
    for iterations in (1, 4):
        X, v = run(cuda, H, k, iterations)
        Xr, vr = reference(H, k, iterations)
        tol = 4 * n * 2.0 ** -53 * (1 / gap).max() * max(D.max(), 1e-300) * np.abs(Xr).max()
        assert np.abs(X - Xr).max() <= tol + 1e-300
        assert np.abs(v - vr).max() <= n * 2.0 ** -52 * np.abs(H).max()


def test_nonfinite_entries_travel_as_in_fp64(cuda):
    """An infinite entry of H gives the Inf / NaN pattern of the FP64 map."""
    rng = np.random.default_rng(3)
    n, k = 200, 20
    H = rng.standard_normal((n, n)) * 0.01
    H[np.arange(n), np.arange(n)] = np.arange(n)
    H[150, 3] = np.inf
    X, _ = run(cuda, H, k, 1)
    d = np.diag(H)
    with np.errstate(invalid="ignore", divide="ignore"):
        E = np.eye(n, k)
        Y = H @ E
        c = np.diagonal(Y[:k]) - d[:k]
        want = (Y - d[:, None] * E - E * c[None, :]) / (d[None, :k] - d[:, None])
    want[np.arange(k), np.arange(k)] = 1.0
    assert (np.isnan(X) == np.isnan(want)).all()
    assert (X[np.isinf(want)] == want[np.isinf(want)]).all()


def test_subnormal_row_scales(cuda):
    """Rows of Delta far below the fast split's range."""
    rng = np.random.default_rng(5)
    n, k = 160, 18
    H = rng.standard_normal((n, n)) * 0.01
    H[40:80] *= 2.0 ** -1000
    H[np.arange(n), np.arange(n)] = np.arange(n)
    X, _ = run(cuda, H, k, 3)
    Xr, _ = reference(H, k, 3)
    # rows 40..79: relative to their own scale, down to the subnormal spacing
    D = np.abs(H - np.diag(np.diag(H)))
    scale = D.max(axis=1)[:, None] * np.abs(Xr).max(axis=0)[None, :]
    assert (np.abs(X - Xr) <= 16 * n * 2.0 ** -53 * scale + 2.0 ** -1070).all()
