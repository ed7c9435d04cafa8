"""Vectors of so few contracted values (up to 64) that the digit kernel finds the
row exponents itself, and one size beyond: one sector of D multiplets and
several, rows of zeros, rows of very different scales, vectors near the largest
and the smallest normal numbers.  The split modes' tolerances: 1e-12 (7 slices)
and 1e-10 (6 slices), relative (Frobenius); a batch of one, which takes the
other way, equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {1: 1e-12, 2: 1e-10}


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("scale", [0, 1000, -900])
@pytest.mark.parametrize("D,nspin1,max2j", [(1, 0, 0), (3, 1, 2), (31, 0, 0), (32, 0, 0), (33, 0, 0), (63, 0, 0), (64, 0, 0),
                                            (65, 0, 0), (100, 4, 12), (200, 3, 10)])
def test_small_rows(su2lib, oracle, mode, scale, D, nspin1, max2j):
    import torch

    from su2dmrg_gb300.su2 import HeffBatch, HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=D, max2j=max2j)
    psi, terms, hl, hr = w.to_device()
    rng = np.random.default_rng(D)
    x = w.psi_data.copy()
    off, _ = w.psi.offsets()
    for b in np.flatnonzero(w.psi.flag):  # rows and columns of one block over 40 binary orders, one row of zeros
        m, n = w.psi.block_shape(b)
        blk = x[off[b]:off[b] + m * n].reshape(m, n, order="F")
        blk = np.ldexp(blk, rng.integers(-20, 21, (m, 1)) + rng.integers(-20, 21, (1, n)))
        if m > 2:
            blk[m // 2] = 0.0
        x[off[b]:off[b] + m * n] = blk.ravel(order="F")
    x /= np.linalg.norm(x)
    prob = oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr)
    ref = oracle.heff_apply(prob, x)
    v = torch.from_numpy(np.ldexp(x, scale)).cuda()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=mode)
    y, z = torch.full_like(psi, float("nan")), torch.full_like(psi, float("nan"))
    plan.apply(v, y)
    HeffBatch([plan]).apply(v, z)
    torch.cuda.synchronize()
    assert plan.status() == 0 and torch.equal(y, z)
    assert np.linalg.norm(np.ldexp(y.cpu().numpy(), -scale) - ref) <= TOL[mode] * np.linalg.norm(ref)
