"""The last group of the 6-slice split GEMM (weight 1/2 of the fixed point's
unit) is kept in full until the sums of a chunk are rounded to the unit.

One square block, y = H_L^T psi, whose only nonzero digit products fall into
that group: H_L has a 1 in row 0 and psi in row 1 (they set every row's
exponent to 2 and meet zeros), and n rows hold 2^-40 (its last digit is 1) in the
one and 2^-5 (its first digit is 1) in the other.  So y = n 2^-45 exactly, the
unit is 2^(2 + 2 - 48) = 2^-44, and the only rounding left is that of each
chunk of 560 rows to a multiple of the unit: at most 2^-45 a chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low_in_psi", [False, True])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("D,n", [(40, 1), (40, 2), (40, 3), (40, 5), (40, 6), (40, 7), (40, 38), (560, 558), (562, 560),
                                 (1124, 1122), (1700, 1698)])
def test_last_group_is_kept(su2lib, D, n, sign, low_in_psi):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=0, seed=1, max2j=0)
    (hs, hx, _), psi = w.hl, w.psi_data
    assert hx.size == psi.size == D * D
    h, p = np.zeros((D, D)), np.zeros((D, D))  # h[column, row], p[column, row]
    h[:, 0], p[:, 1] = 1.0, 1.0
    h[:, 2: 2 + n], p[:, 2: 2 + n] = sign * 2.0**-40, 2.0**-5
    if low_in_psi:
        h[:, 2: 2 + n], p[:, 2: 2 + n] = 2.0**-5, sign * 2.0**-40
    plan = HeffPlan(w.psi, [], (hs, torch.from_numpy(h.ravel()).cuda(), 1.0), None, mode=2)
    x = torch.from_numpy(p.ravel()).cuda()
    y = torch.full_like(x, float("nan"))
    plan.apply(x, y)
    torch.cuda.synchronize()
    assert plan.status() == 0
    chunks = -(-(2 + n) // 560)
    assert np.abs(y.cpu().numpy() - sign * n * 2.0**-45).max() <= chunks * 2.0**-45
