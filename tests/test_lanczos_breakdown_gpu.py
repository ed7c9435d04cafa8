"""Lanczos started in an invariant subspace of k dimensions: the residual norm
vanishes at step k, also where the coefficients are not read at that step, and
the solve ends there: the matvecs counted are the k steps, the check at step 4
if it was passed, and the final check.  The energy is the lowest eigenvalue of
the subspace (to 1e-12 of the spectrum's width, rounding of a few dozen
products), the vector its eigenvector.  Solving again with the same plan, by
captured steps, gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7])
def test_invariant_subspace(su2lib, mode, k):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=6, nspin1=1, seed=5, max2j=2)
    psi, terms, hl, hr = w.to_device()
    n = psi.numel()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=mode)
    h = np.zeros((n, n))
    y = torch.empty_like(psi)
    for i in range(n):
        e = torch.zeros_like(psi)
        e[i] = 1.0
        plan.apply(e, y)
        h[:, i] = y.cpu().numpy()
    ev, vec = np.linalg.eigh(0.5 * (h + h.T))
    assert np.abs(h - h.T).max() <= 1e-12 * np.abs(ev).max()
    pick = np.linspace(0, n - 1, k).round().astype(int)
    start = vec[:, pick].sum(axis=1) / np.sqrt(k)
    got = []
    for _ in range(3):
        x = torch.from_numpy(start.copy()).cuda()
        energy, matvecs = plan.lanczos(x, mlanc=30)
        got.append((energy, matvecs, x.cpu().numpy()))
    energy, matvecs, v = got[0]
    assert matvecs == k + (1 if k > 4 else 0) + 1
    assert abs(energy - ev[pick[0]]) <= 1e-12 * np.abs(ev).max()
    assert abs(abs(v @ vec[:, pick[0]]) - 1) <= 1e-10
    for other in got[1:]:
        assert other[0] == energy and other[1] == matvecs and (other[2] == v).all()
