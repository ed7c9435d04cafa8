"""The split GEMM at block sizes around its tile's warp edges (32 rows, 16
columns, 128 x 64), where whole warps of a tile lie beyond the block: one
sector of D multiplets, square products.  The split modes' tolerances: 1e-12
(7 slices) and 1e-10 (6 slices), relative (Frobenius)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {1: 1e-12, 2: 1e-10}


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("D", [2, 14, 18, 31, 32, 34, 47, 48, 50, 63, 66, 95, 96, 98, 111, 112, 114, 127, 128, 130, 160,
                               162, 193, 257])
def test_block_edges(su2lib, oracle, mode, D):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=0, seed=D, max2j=0)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=mode)
    y = torch.full_like(psi, float("nan"))
    plan.apply(psi, y)
    torch.cuda.synchronize()
    assert plan.status() == 0
    ref = oracle.heff_apply(oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr), w.psi_data)
    assert np.linalg.norm(y.cpu().numpy() - ref) <= TOL[mode] * np.linalg.norm(ref)
