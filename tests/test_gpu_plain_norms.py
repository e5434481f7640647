"""The step norms of a tolerance-stopped plain solve, which reach the host with
the next step or, where none follows, from a kernel of their own: limits of
one step to more than are needed, a tolerance met at once, one or several
update blocks."""
import numpy as np
import pytest

from block_ipt_gb300 import api
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(30, 1), (256, 8), (300, 40), (1100, 3)])
@pytest.mark.parametrize("maxiter,tol", [(1, 1e-30), (2, 1e-30), (3, 1e-30), (7, 1e-30),
                                         (50, 0.5), (50, 1e-12)])
def test_steps_and_residual_as_the_oracle(cuda, n, k, maxiter, tol):
    """The residual is ||X' - X|| / ||X||; both norms carry the rounding of the
    step, 1e-13 of ||X||, and of their sums, 1e-13 of themselves."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) * (0.05 / np.sqrt(n))
    H = np.asfortranarray(A + A.T + np.diag(np.arange(1.0, n + 1)))
    X, v, info = api.ipt_cuda_tol(H, k, tol, maxiter)
    it, res = info["iterations"], info["fixed_point_residual"]
    Xo, vo, ito, reso = oracle.ipt_dense(H, k, maxiter, tol, True)
    assert it == ito
    assert abs(res - reso) <= 1e-13 + 1e-13 * reso
    assert np.abs(X - Xo).max() <= 1e-12
    assert np.abs(v - vo).max() <= 1e-12 * n
