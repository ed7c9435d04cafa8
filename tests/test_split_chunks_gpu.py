"""The split GEMM at the segment lengths where its chunks and stages change:
fewer K stages than the low groups run ahead, as many, one more; one stage
below, at and above the 35 of a chunk; two chunks and more.  One sector of D
multiplets makes every product of the plan a D x D x D one.  The split modes'
tolerances: 1e-12 (7 slices) and 1e-10 (6 slices), relative (Frobenius).

And vectors near the smallest normal number, whose results are subnormal: the
same tolerance plus what rounding the intermediates and the result to multiples
of 2^-1074 allows (an intermediate's half unit, times a column of an operator
of norm about 1, is below a unit; 64 units leave room)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {1: 1e-12, 2: 1e-10}


def _plan(D, nspin1, mode, seed, max2j):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=seed, max2j=max2j)
    psi, terms, hl, hr = w.to_device()
    return torch, w, psi, HeffPlan(w.psi, terms, hl, hr, mode=mode)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("D", [1, 15, 16, 17, 33, 49, 64, 65, 80, 81, 544, 545, 560, 561, 577, 625, 1121])
def test_chunk_lengths(su2lib, oracle, mode, D):
    torch, w, psi, plan = _plan(D, 0, mode, D, 0)
    y = torch.full_like(psi, float("nan"))
    plan.apply(psi, y)
    torch.cuda.synchronize()
    assert plan.status() == 0
    ref = oracle.heff_apply(oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr), w.psi_data)
    assert np.linalg.norm(y.cpu().numpy() - ref) <= TOL[mode] * np.linalg.norm(ref)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("D,nspin1,max2j", [(40, 0, 0), (90, 2, 4)])
def test_subnormal_results(su2lib, oracle, mode, D, nspin1, max2j):
    torch, w, psi, plan = _plan(D, nspin1, mode, 3, max2j)
    tiny = np.ldexp(w.psi_data / np.abs(w.psi_data).max(), -1016)
    y = torch.full_like(psi, float("nan"))
    plan.apply(torch.from_numpy(tiny).cuda(), y)
    torch.cuda.synchronize()
    assert plan.status() == 0
    prob = oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr)
    ref = oracle.heff_apply(prob, np.ldexp(tiny, 1000))  # exact scaling of the very inputs
    got = np.ldexp(y.cpu().numpy(), 1000)
    assert 0 < np.count_nonzero(np.abs(y.cpu().numpy()) < 2.0**-1022)
    assert np.linalg.norm(got - ref) <= TOL[mode] * np.linalg.norm(ref) + 64 * 2.0**-74 * np.sqrt(ref.size)
