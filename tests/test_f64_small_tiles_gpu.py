"""The FP64 engine where its launch tiles are 16 x 16 (short single products
that leave 32 x 32 tiles uneven) or 8 x 8 with a split contraction of few
values: systems of a handful of multiplets up to the sizes where 32 x 32 tiles
take over.  Tolerance: sums over at most a few thousand products of entries of
one scale round to about 2e-14 relative (Frobenius); 1e-13."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,nspin1,max2j,spin0", [
    (2, 1, 1, False), (4, 1, 2, True), (8, 4, 12, True), (16, 2, 12, False), (24, 2, 12, True), (24, 6, 6, True),
    (60, 3, 12, False), (123, 5, 10, True), (150, 6, 9, True), (200, 6, 12, False), (230, 9, 12, True),
    (270, 9, 12, True)])
def test_small_heff(su2lib, oracle, D, nspin1, max2j, spin0):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=D + 1, max2j=max2j, spin0=spin0)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=0)
    y = torch.full_like(psi, float("nan"))
    plan.apply(psi, y)
    torch.cuda.synchronize()
    ref = oracle.heff_apply(oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr), w.psi_data)
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-13 * np.linalg.norm(ref)
