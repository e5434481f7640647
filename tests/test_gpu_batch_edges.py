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


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_estimated_launch_shape_matches_single_cta(cuda, monkeypatch, precision):
    """The launch shape picked by the estimated schedule gives the blocks and
    sweep counts of one CTA per instance."""
    torch = cuda
    rng = np.random.default_rng(3)
    specs = [(int(rng.integers(64, 420)), int(rng.integers(1, 17))) for _ in range(90)]
    results = {}
    for pct in (None, "0"):
        if pct is None:
            monkeypatch.delenv("IPT_GB300_BATCH_TEAM_PCT", raising=False)
        else:
            monkeypatch.setenv("IPT_GB300_BATCH_TEAM_PCT", pct)
        keep, inst = [], []
        for s, (n, k) in enumerate(specs):
            H, _ = workloads.batch_instance(n, 0.05, 400 + s)
            dH = torch.from_numpy(np.asfortranarray(H).T.copy()).cuda()
            dX = torch.zeros((k, n), dtype=torch.float64, device="cuda")
            dv = torch.zeros(k, dtype=torch.float64, device="cuda")
            keep.append((dH, dX, dv))
            inst.append((dH.data_ptr(), n, k, dX.data_ptr(), dv.data_ptr()))
        plan = api.BatchPlan(inst, precision)
        assert plan.shape()["cluster"] in ((1, 2, 4, 8) if pct is None else (1,))
        plan.run()
        torch.cuda.synchronize()
        results[pct] = [(dX.cpu().numpy(), rep["iterations"], rep["converged"])
                        for (_, dX, _), rep in zip(keep, plan.reports())]
        plan.close()
    for (Xa, ia, ca), (Xb, ib, cb) in zip(results[None], results["0"]):
        assert ca == 1 and cb == 1 and ia == ib
        assert np.abs(Xa - Xb).max() <= 1e-12
