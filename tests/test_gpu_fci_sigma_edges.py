"""The matrix-free sigma at the edges of its coupling loop (fewer than 32
couplings per row, remainders, one beta single per string) against the CPU
restatement, to the FP64 rounding of the sums (about 1e-15 per term, at most
a few hundred terms: 1e-13 of the largest entry)."""
import numpy as np
import pytest

from block_ipt_gb300 import api
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,na,nb", [(2, 1, 1), (3, 1, 2), (3, 2, 1), (4, 2, 1), (5, 2, 3),
                                        (6, 1, 5), (7, 3, 4)])
@pytest.mark.parametrize("k", [1, 8, 9])
def test_sigma(cuda, norb, na, nb, k):
    torch = cuda
    spec = api.fci_spec(norb, na, nb, seed=4)
    n = api.fci_dimension(spec)
    X = np.random.default_rng(n).standard_normal((n, k))
    dX = torch.from_numpy(X.T.copy()).cuda()
    dY = torch.empty((k, n), dtype=torch.float64, device="cuda")
    api.fci_sigma(spec, dX.data_ptr(), k, dY.data_ptr(), "fp64")
    ref = oracle.fci_sigma(norb, na, nb, X, seed=4)
    assert np.abs(dY.T.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
