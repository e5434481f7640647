"""Gradient of the learned preconditioner at the edges of its launch shapes:
single rows, 128-row tiles with remainders, one tile per SM, several tiles per
CTA; against the CPU oracle in float64.

Tolerance: FP32 forward and backward passes (a few hundred operations of unit
roundoff 6e-8 per entry) and FP32 sums over at most ~1e4 terms whose rounding
errors are random: 1e-4 of the largest entry of each parameter block."""
import numpy as np
import pytest

from block_ipt_gb300 import api
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 129, 1000, 19456, 19457, 60001])
def test_gradient(cuda, rows):
    torch = cuda
    rng = np.random.default_rng(rows)
    P = torch.empty(api.mlp_param_count(), dtype=torch.float32, device="cuda")
    api.mlp_init(P.data_ptr(), 5)
    P[4608:4672] = torch.from_numpy(rng.standard_normal(64).astype(np.float32) * 0.3).cuda()
    data = np.column_stack([rng.standard_normal((rows, 7)), rng.uniform(0.1, 2.0, rows)])
    data = data.astype(np.float32)
    # one float of offset: rows of any 4-byte alignment are accepted
    buf = torch.zeros(8 * rows + 1, dtype=torch.float32, device="cuda")
    buf[1:] = torch.from_numpy(data.reshape(-1)).cuda()
    g = torch.empty(api.mlp_param_count() + 1, dtype=torch.float32, device="cuda")
    api.mlp_loss_grad(P.data_ptr(), buf.data_ptr() + 4, rows, g.data_ptr())
    g = g.cpu().numpy().astype(np.float64)
    loss, ref = M.loss_grad(P.cpu().numpy(), data)
    assert abs(g[-1] - loss) <= 1e-5 * max(1.0, loss)
    for lo, hi in [(0, 384), (384, 448), (448, 4544), (4544, 4608), (4608, 4672), (4672, 4673)]:
        assert np.abs(g[lo:hi] - ref[lo:hi]).max() <= 1e-4 * max(np.abs(ref[lo:hi]).max(), 1e-8)
