"""Davidson solves whose block products run in double-float arithmetic or on
the FP64 pipe, at the edges of those kernels' tiles: blocks of one column to
more than 16 (the Gram tiles are 8, 16 and 32 wide, the tall products 4, 8 and
16, the sparse product 4, 8 and 16), a row count below, at and past the 32-row and 128-row stages,
rows with fewer nonzeros than one round of the sparse product takes, exact
zeros, and restarts of a small basis."""
import numpy as np
import pytest

from block_ipt_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 129, 1000])
@pytest.mark.parametrize("k,max_basis", [(1, 4), (3, 12), (5, 0), (8, 32), (13, 40), (17, 60),
                                         (33, 100)])
@pytest.mark.parametrize("df", ["0", "1"])
def test_davidson_products_at_tile_edges(cuda, monkeypatch, df, n, k, max_basis):
    """Bounds of the solver: eigenvalues within 1e-10 ||H||, residuals 1e-8."""
    from scipy.sparse import csr_matrix, random as sprandom
    if 2 * k > n:
        pytest.skip("needs a basis smaller than the space")
    monkeypatch.setenv("IPT_GB300_DF_DAVIDSON", df)
    rng = np.random.default_rng(100 * k + n)
    A = sprandom(n, n, density=min(0.2, 12.0 / n), random_state=rng, format="csr") * 0.05
    d = np.arange(n) * 0.5 + rng.uniform(0, 0.1, n)
    H = (A + A.T + csr_matrix((d, (np.arange(n), np.arange(n))), shape=(n, n))).tocsr()
    H.sort_indices()
    X, v, rep = api.block_solve_csr(H.indptr, H.indices, H.data, n, k, "fp64", strategy=1,
                                    max_basis=max_basis)
    Hd = H.toarray()
    hn = np.abs(Hd).sum(axis=1).max()
    assert rep["converged"] == 1
    assert np.abs(v - np.linalg.eigvalsh(Hd)[:k]).max() <= 1e-10 * hn
    assert np.abs(np.linalg.norm(X, axis=0) - 1.0).max() <= 1e-10
    assert np.linalg.norm(Hd @ X - X * v, axis=0).max() <= 1e-8 * max(1.0, hn)
