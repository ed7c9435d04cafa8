"""The Lanczos solve where its vectors go through one cluster: one square block,
so D^2 elements, from one element to the longest vector a cluster takes (16,384)
and one size beyond, either side of every number of elements a thread, with
idle CTAs (short vectors) and a last CTA that holds fewer; the shortest
recurrences, more Krylov vectors than one combination takes.  The bounds of
the suite's Lanczos tests: energy within 1e-10 relative of the oracle's
lanczos1, the same number of matvecs, overlap 1 to 1e-9, and a batch of one
equal to the solo solve bit for bit, also when it runs as captured steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,mlanc", [(3, 3), (4, 2), (11, 5), (44, 5), (45, 5), (46, 5), (64, 4), (65, 9), (90, 5), (91, 21),
                                     (127, 3), (128, 5), (129, 5)])
def test_square_block(su2lib, oracle, D, mlanc):
    import torch

    from su2dmrg_gb300.su2 import HeffBatch, HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=0, seed=D, max2j=0)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=0)
    got = []
    for _ in range(3):
        v = psi.clone()
        e, nmv = plan.lanczos(v, mlanc=mlanc)
        got.append((e, nmv, v))
    b = psi.clone()
    (eb, nb), = HeffBatch([plan]).lanczos([b], mlanc=mlanc)
    got.append((eb, nb, b))
    e, nmv, v = got[0]
    for other in got[1:]:
        assert other[:2] == (e, nmv) and torch.equal(other[2], v)
    prob = oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr)
    e_or, v_or, nmv_or = oracle.lanczos1(lambda x: oracle.heff_apply(prob, x), w.psi_data.copy(), mlanc)
    assert abs(e - e_or) <= 1e-10 * abs(e_or)
    assert nmv == nmv_or
    x = v.cpu().numpy()
    assert abs(abs(x @ v_or) / (np.linalg.norm(x) * np.linalg.norm(v_or)) - 1) <= 1e-9
