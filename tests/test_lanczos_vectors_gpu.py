"""The Lanczos solve's vector kernels at the lengths where they change: vectors
shorter than one block of threads, a few blocks, and long enough for four
elements a thread at a time; the shortest recurrences, ones that pass the
convergence check, and more Krylov vectors than one combination launch takes.
Energy within 1e-10 relative of the oracle's lanczos1 (the suite's bound), the
same number of matvecs, the same vector (overlap 1 to 1e-9: both sides stop on
an overlap known to 1e-8), and a batch of one equal to the solo solve bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,nspin1,mlanc,max2j", [
    (3, 1, 2, 1), (5, 1, 3, 2), (12, 2, 5, 2), (30, 2, 4, 4), (60, 3, 9, 6), (60, 3, 21, 6), (1300, 1, 3, 12)])
def test_lanczos_lengths(su2lib, oracle, D, nspin1, mlanc, max2j):
    import torch

    from su2dmrg_gb300.su2 import HeffBatch, HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=D, max2j=max2j)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=0)
    v = psi.clone()
    e, nmv = plan.lanczos(v, mlanc=mlanc)
    b = psi.clone()
    batch = HeffBatch([plan])
    (eb, nb), = batch.lanczos([b], mlanc=mlanc)
    assert (eb, nb) == (e, nmv) and torch.equal(v, b)
    prob = oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr)
    e_or, v_or, nmv_or = oracle.lanczos1(lambda x: oracle.heff_apply(prob, x), w.psi_data.copy(), mlanc)
    assert abs(e - e_or) <= 1e-10 * abs(e_or)
    assert nmv == nmv_or
    got = v.cpu().numpy()
    assert abs(abs(got @ v_or) / (np.linalg.norm(got) * np.linalg.norm(v_or)) - 1) <= 1e-9
