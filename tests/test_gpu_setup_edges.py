"""The dense setup pass of the mixed solves on inputs that take its side
branches: a column maximum that is a power of two (the scale then depends on
the low word too), exact zeros and entries far below a float's remainder, the
diagonal in either half of a pair, odd and ragged sizes, large and small
scales."""
import numpy as np
import pytest

from block_ipt_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 65, 257, 514, 1030])
@pytest.mark.parametrize("kind", ["powers", "zeros", "tiny", "scaled"])
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
def test_setup_side_branches(cuda, n, kind, precision):
    """The norm is summed with 48 bits an entry (n 2^-48); the pairs meet the
    solver's bounds (eigenvalues 1e-10 ||H||, residuals 1e-8)."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) * 0.01 / np.sqrt(n)
    A = A + A.T
    if kind == "powers":
        A = np.sign(A) * 2.0 ** np.floor(np.log2(np.abs(A)))
    elif kind == "zeros":
        A[np.abs(A) < np.quantile(np.abs(A), 0.7)] = 0.0
    elif kind == "tiny":
        small = np.abs(A) < np.quantile(np.abs(A), 0.5)
        A[small] *= 2.0 ** -80
        A[np.abs(A) < np.quantile(np.abs(A), 0.1)] *= 2.0 ** -120
    A = np.triu(A, 1)
    d = np.arange(1, n + 1) * 0.5
    H = A + A.T + np.diag(d)
    if kind == "scaled":
        H = H * 2.0 ** 30
    k = 6
    X, v, rep = api.block_solve_dense(np.asfortranarray(H), k, precision)
    hn = np.abs(H).sum(axis=1).max()
    assert rep["converged"] == 1
    assert abs(rep["matrix_norm_inf"] - hn) <= n * 2.0 ** -48 * hn
    assert np.abs(v - np.linalg.eigvalsh(H)[:k]).max() <= 1e-10 * hn
    assert np.linalg.norm(H @ X - X * v, axis=0).max() <= 1e-8 * max(1.0, hn)
