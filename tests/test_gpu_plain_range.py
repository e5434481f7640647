"""Entries of very different size in the plain FP64 path (ipt_cuda_device,
acx_cuda_device_tol, the block solver's FP64 solve).  Rows whose entries span
many binades within 128 columns are multiplied in FP64 FMAs, entry by entry as
accurate as FP64 is; all others on the tensor cores, in 56-bit fixed point per
block of 128 columns, however far the blocks lie apart.

Tolerances.  FP64 FMAs: tests/test_gpu_fp64_fma.py.  Tensor cores: a block of m
columns adds at most m 2^-54 (1 + 2^-5) max|Delta_il| max|X_lc| to the error of
an entry of Delta X (each operand is cut off below 2^-56 of the next power of
two above its block's largest; the dropped digit products and the alignment of
the blocks stay below 2^-59 of it), the sum and the map eight roundings; one
step's error travels through the next as the map's derivative does.
"""
import numpy as np
import pytest

from block_ipt_gb300 import _lib, api
from tests.test_gpu_fp64_fma import acx, fixed_point, graded, plain

pytestmark = pytest.mark.gpu

B = 128


def with_diagonal(D, d):
    H = np.array(D)
    H[np.arange(len(d)), np.arange(len(d))] = d
    return H


def noise(n, seed):
    A = np.triu(np.random.default_rng(seed).standard_normal((n, n)), 1)
    return A + A.T


def decaying(n, length, seed):
    i = np.arange(n)
    rng = np.random.default_rng(seed + 1)
    return with_diagonal(0.05 * noise(n, seed) * np.exp(-np.abs(i[:, None] - i[None, :]) / length),
                         i + 0.5 * rng.uniform(size=n))


def tridiagonal(n, seed):
    i = np.arange(n)
    return with_diagonal(0.05 * noise(n, seed) * (np.abs(i[:, None] - i[None, :]) <= 1), i + 0.0)


def permuted(H, seed):
    p = np.random.default_rng(seed).permutation(len(H))
    return H[np.ix_(p, p)]


def block_scaled(n, decades, seed):
    """Every block of 128 columns `decades` above (below) the one before."""
    s = 10.0 ** (decades * (np.arange(n) // B))
    return with_diagonal(noise(n, seed) * (0.1 / n) * (s / s.max())[None, :], np.arange(n) + 0.0)


def block_diagonal(n, seed):
    b = np.arange(n) // B
    return with_diagonal(noise(n, seed) * (0.2 / B) * (b[:, None] == b[None, :]), np.arange(n) + 0.0)


def split_iterates(H, k, steps):
    """(t, the map's iterate after t steps in extended precision, a bound of
    the split product's error) for the first and the last step."""
    n = len(H)
    d = np.diag(H)
    D = np.abs(H - np.diag(d))
    gap = np.abs(d[None, :k] - d[:, None])
    gap[np.arange(k), np.arange(k)] = np.inf
    starts = np.arange(0, n, B)
    m = np.diff(np.append(starts, n))
    R = np.maximum.reduceat(D, starts, axis=1)
    u = 2.0 ** -53
    X, err = np.eye(n, k, dtype=np.longdouble), np.zeros((n, k))
    for t in range(1, steps + 1):
        A = np.abs(X).astype(np.float64) + err
        X = fixed_point(H, k, 1, X)
        prod = (R * (m * (1 + 2.0 ** -5) * u / 2)[None, :]) @ np.maximum.reduceat(A, starts, axis=0)
        prod += D @ err
        Y = D @ A
        c, dc = np.diagonal(Y[:k]), np.diagonal(prod[:k])
        err = (prod + err * c[None, :] + A * dc[None, :] + 8 * u * (Y + A * c[None, :])) / gap
        err += 8 * u * np.abs(X).astype(np.float64)
        if t in (1, steps):
            yield t, X, err


SPLIT = {"decay64": lambda n: decaying(n, 64.0, 3), "gauss": lambda n: block_scaled(n, 0, 4),
         "up": lambda n: block_scaled(n, 30, 5), "down": lambda n: block_scaled(n, -30, 6),
         "up9": lambda n: block_scaled(n, 9, 7), "blocks": lambda n: block_diagonal(n, 8)}


@pytest.mark.parametrize("family", sorted(SPLIT))
@pytest.mark.parametrize("n,k", [(129, 5), (300, 17), (700, 33), (1025, 9)])
def test_entries_of_the_split_product(cuda, family, n, k):
    H = SPLIT[family](n)
    for steps, Xr, tol in split_iterates(H, k, 3):
        X = plain(cuda, H, k, steps)
        assert (np.abs(X - Xr) <= tol + 1e-300).all()


WIDE = {"graded12": lambda n: graded(n, 12, 1), "graded20": lambda n: graded(n, 20, 1),
        "decay16": lambda n: decaying(n, 16.0, 3)}


@pytest.mark.parametrize("family", sorted(WIDE))
def test_entries_of_wide_rows(cuda, family):
    n, k = 300, 8
    H = WIDE[family](n)
    for steps in (1, 12):
        X = plain(cuda, H, k, steps)
        Xr = fixed_point(H, k, steps)
        if family == "decay16":
            # the diagonal carried through (d |X|) and the sums of magnitudes,
            # both relative to an entry, carried on by a contracting map
            D = np.abs(H - np.diag(np.diag(H)))
            d = np.diag(H)
            gap = np.abs(d[None, :k] - d[:, None])
            gap[np.arange(k), np.arange(k)] = np.inf
            size = (D @ np.abs(Xr) + d[:, None] * np.abs(Xr)) / gap
            tol = 16 * n * 2.0 ** -53 * size
            assert (np.abs(X - Xr) <= tol).all()
        else:
            assert (np.abs(X - Xr) <= 16 * n * 2.0 ** -53 * np.abs(Xr)).all()
    if family != "decay16":
        Xr = fixed_point(H, k, 40)
        assert (np.abs(acx(cuda, H, k) - Xr) <= 16 * n * 2.0 ** -53 * np.abs(Xr)).all()


ROUTES = [("decay64", SPLIT["decay64"], False), ("gauss", SPLIT["gauss"], False),
          ("up", SPLIT["up"], False), ("blocks", SPLIT["blocks"], False),
          ("graded20", lambda n: graded(n, 60, 1), True),
          ("permuted", lambda n: permuted(graded(n, 20, 1), 2), True),
          ("decay16", WIDE["decay16"], True), ("tridiagonal", lambda n: tridiagonal(n, 2), True)]


@pytest.mark.parametrize("name,family,wide", ROUTES, ids=[r[0] for r in ROUTES])
def test_route(cuda, name, family, wide):
    n, k = 1100, 4
    H = family(n)
    lib = _lib.load()
    counts = []
    for steps in (2, 10):
        before = lib.ipt_block_launch_count()
        plain(cuda, H, k, steps)
        counts.append(lib.ipt_block_launch_count() - before)
    # digits, product and update, or product and update
    assert counts[1] - counts[0] == 8 * (2 if wide else 3)


def test_block_solve_of_a_wide_matrix(cuda):
    n, k = 900, 6
    H = tridiagonal(n, 4)
    dH = cuda.from_numpy(H).cuda()
    X = cuda.empty(k, n, dtype=cuda.float64, device="cuda")
    w = cuda.empty(k, dtype=cuda.float64, device="cuda")
    api.block_solve_dense_device(dH.data_ptr(), n, k, X.data_ptr(), w.data_ptr(), "fp64")
    # eigenvalues to the solver's residual tolerance
    assert np.abs(w.cpu().numpy() - np.linalg.eigvalsh(H)[:k]).max() <= 1e-10 * np.abs(H).sum(1).max()
