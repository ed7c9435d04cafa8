"""Split-precision output tiles summed from partial tiles (reduce_partials): few
and many parts per tile, counts that are and are not multiples of the four
loads a thread keeps in flight, blocks smaller than a tile and ragged ones.
The 7-slice tolerance of the split mode, 1e-12 relative (Frobenius) against
the FP64 oracle, and the same bits on a second application."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,nspin1,max2j", [(9, 1, 2), (24, 2, 4), (40, 5, 6), (131, 3, 12), (150, 13, 8), (333, 4, 3)])
def test_partial_sums_match_oracle(su2lib, oracle, D, nspin1, max2j):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=D, max2j=max2j)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=1)
    y, y2 = (torch.full_like(psi, float("nan")) for _ in range(2))
    plan.apply(psi, y)
    plan.apply(psi, y2)
    torch.cuda.synchronize()
    assert plan.status() == 0
    ref = oracle.heff_apply(oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr), w.psi_data)
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)
    assert torch.equal(y, y2)
