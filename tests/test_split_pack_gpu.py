"""The digit pack where it can go wrong: operands of any row scale and either
storage order, coefficients +1, -1 and others, rows and k that end inside a
group, a tile or a chunk.

A power of two on a row of an operand moves only that row's exponent, so the
result's rows (or columns) move by exactly that power: bit for bit while the
scaling goes through the multiply-add (exponents up to about 2^951), and within
the split mode's tolerance of 1e-12 a row beyond, where rows are scaled by
integer shifts (another rule for ties)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coef", [1.0, -1.0, 0.3])
@pytest.mark.parametrize("side", ["hl", "hr"])
@pytest.mark.parametrize("D,top", [(7, 900), (70, 900), (157, 900), (301, 900), (70, 1000)])
def test_row_scales(su2lib, side, D, top, coef):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=0, seed=D, max2j=0)
    psi, _terms, hl, hr = w.to_device()
    s, x, _ = hl if side == "hl" else hr
    k = np.random.default_rng(5).integers(-top, top + 1, D)
    k[:2] = top, -top

    def run(data):
        h = (s, data, coef)
        plan = HeffPlan(w.psi, [], h if side == "hl" else None, h if side == "hr" else None, mode=1)
        y = torch.full_like(psi, float("nan"))
        plan.apply(psi, y)
        torch.cuda.synchronize()
        assert plan.status() == 0
        return y.cpu().numpy().reshape(D, D)  # [column, row] of the one column-major block

    # y = coef H_L^T psi takes its row i from H_L's column i, y = coef psi H_R its column i from H_R's
    # (numpy's ldexp is exact; torch's multiplies by a computed power)
    scaled = torch.from_numpy(np.ldexp(x.cpu().numpy().reshape(D, D), k[:, None]).ravel()).cuda()
    base, got = run(x), run(scaled)
    want = np.ldexp(base, k[None, :] if side == "hl" else k[:, None])
    if top <= 900:
        assert np.array_equal(got, want)
    else:
        scale = np.abs(want).max(axis=0 if side == "hl" else 1, keepdims=True)
        assert (np.abs(got - want) <= 1e-12 * scale).all()
