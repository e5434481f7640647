"""The ACX map divides by d_c - d_i with one rounding, as the reference does
(IPT_C_GPU/src/ACX/acx_cuda.cu:109-172).  Couplings of 53 bits within one
binade are exact in the product's fixed point, and so small that the first
evaluation F(I) = Delta_ic / (d_c - d_i) is the result: its entries are the
correctly rounded quotients."""
import numpy as np
import pytest

from tests.test_gpu_acx import run_acx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(40, 7), (300, 20), (1100, 40)])
@pytest.mark.parametrize("knob", [None, "IPT_GB300_FP64_DFMA"])
def test_quotients_are_correctly_rounded(cuda, monkeypatch, n, k, knob):
    if knob is not None:
        monkeypatch.setenv(knob, "1")
    rng = np.random.default_rng(n)
    A = np.triu(1 + rng.uniform(size=(n, n)), 1) * 2.0 ** -50
    d = np.cumsum(1 + rng.uniform(size=n))
    H = A + A.T
    H[np.arange(n), np.arange(n)] = d
    den = d[None, :k] - d[:, None]
    den[np.arange(k), np.arange(k)] = 1
    want = (A + A.T)[:, :k] / den
    want[np.arange(k), np.arange(k)] = 1
    status, X, _, info = run_acx(cuda, H, k, 1e-12, 5)
    assert status == 0 and info["f_calls"] == 1 and info["converged"] == 1
    assert np.array_equal(X, want)
