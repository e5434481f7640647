"""The FP32 stage of the projected eigensolver at the edges of its pieces: the
bisection takes four eigenvalues per CTA, and the inverse iteration remembers
row exchanges in words of 32 rows."""
import ctypes as C

import numpy as np
import pytest

from block_ipt_gb300 import _lib

pytestmark = pytest.mark.gpu


def run(torch, T):
    m = T.shape[0]
    dT = torch.from_numpy(T).cuda()
    dw = torch.empty(m, dtype=torch.float64, device="cuda")
    dZ = torch.empty((m, m), dtype=torch.float64, device="cuda")
    st = _lib.load().ipt_block_symmetric_eig(C.c_void_p(dT.data_ptr()), m,
                                             C.c_void_p(dw.data_ptr()), C.c_void_p(dZ.data_ptr()),
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    return dw.cpu().numpy(), dZ.T.cpu().numpy()


@pytest.mark.parametrize("m", [3, 4, 5, 31, 32, 33, 34, 63, 64, 65, 66, 95, 97, 98, 111])
@pytest.mark.parametrize("kind", ["exchanges", "no_exchanges"])
def test_tridiagonal_at_word_edges(cuda, m, kind):
    """Tridiagonal inputs: a small diagonal beside large couplings exchanges a
    row in nearly every elimination step, a dominant diagonal in few.  The
    bounds are those of the FP64 polish that follows, 1e-13 ||T||."""
    rng = np.random.default_rng(m)
    d = rng.uniform(-0.1, 0.1, m) if kind == "exchanges" else np.arange(m) * 1.0
    e = rng.uniform(0.5, 1.0, m - 1) * (1.0 if kind == "exchanges" else 0.05)
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    w, Z = run(cuda, T)
    nrm = np.abs(T).sum(axis=1).max()
    assert np.abs(w - np.linalg.eigvalsh(T)).max() <= 1e-13 * nrm
    assert np.abs(Z.T @ Z - np.eye(m)).max() <= 1e-13
    assert np.abs(T @ Z - Z * w).max() <= 1e-12 * nrm
