"""Batched solves at the edges of the double-float sweep's layout: odd and even
column counts (X is staged in pairs of columns), one column, rows just below,
at and past a warp and a 512-row block."""
import numpy as np
import pytest

from block_ipt_gb300 import api, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("threads", [128, 512])
def test_batch_column_pairs_and_row_edges(cuda, precision, threads):
    """Bounds of the batch: residuals 1e-8, eigenvalues within 1e-10 ||H||."""
    torch = cuda
    specs = [(33, 1), (63, 2), (64, 3), (65, 13), (127, 4), (513, 15), (1025, 6), (40, 11)]
    Hs, keep, inst = [], [], []
    for s, (n, k) in enumerate(specs):
        H, _ = workloads.batch_instance(n, 0.05, 40 + s)
        dH = torch.from_numpy(np.asfortranarray(H).T.copy()).cuda()
        dX = torch.zeros((k, n), dtype=torch.float64, device="cuda")
        dv = torch.zeros(k, dtype=torch.float64, device="cuda")
        Hs.append(H)
        keep.append((dH, dX, dv))
        inst.append((dH.data_ptr(), n, k, dX.data_ptr(), dv.data_ptr()))
    plan = api.BatchPlan(inst, precision, threads=threads)
    plan.run()
    torch.cuda.synchronize()
    for (n, k), H, (_, dX, dv), rep in zip(specs, Hs, keep, plan.reports()):
        assert rep["converged"] == 1
        X, v = dX.T.cpu().numpy(), dv.cpu().numpy()
        hn = np.abs(H).sum(axis=1).max()
        r = np.linalg.norm(H @ X - X * v, axis=0) / np.linalg.norm(X, axis=0)
        assert r.max() <= 1e-8 * max(1.0, hn)
        assert np.abs(np.sort(v) - np.linalg.eigvalsh(H)[:k]).max() <= 1e-10 * hn
    plan.close()
