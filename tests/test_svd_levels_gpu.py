"""The truncation's refinement levels, resolved from the basis at hand or by an
eigendecomposition, on one sector of known singular values: fast and slow
decay, values down to the rounding noise, exact and near degeneracies (pairs
and clusters), two groups decades apart, and sectors of one to a few hundred
rows; everything kept, and half.

Bounds: the new V is orthonormal to 1e-13 and U = psi V; the largest half of
the singular values lies within the Gram method's own accuracy of the exact
ones (1e-12 s_max + 1e-15 s_max^2 / s, the bound the truncation's parity tests
use), and where every value is kept and all lie above the noise, U V^T
reconstructs the vector to 1e-13."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECTRA = {
    "decay18": lambda k, n: np.exp(-18.0 * k / n),
    "decay40": lambda k, n: np.exp(-40.0 * k / n),
    "power": lambda k, n: 1.0 / (1.0 + k),
    "pairs": lambda k, n: np.exp(-14.0 * (k // 2) * 2 / n),
    "near": lambda k, n: np.exp(-14.0 * (k // 2) * 2 / n) * (1 + 1e-11 * (k % 2)),
    "clusters": lambda k, n: np.exp(-14.0 * (k // 8) * 8 / n) * (1 + 1e-13 * (k % 8)),
    "two groups": lambda k, n: np.where(k < n // 2, 1 - 0.5 * k / n, 1e-6 * (1 - 0.5 * k / n)),
    "one value": lambda k, n: np.ones(n),
}


@pytest.mark.parametrize("n", [1, 2, 3, 17, 64, 130, 257])
@pytest.mark.parametrize("kind", sorted(SPECTRA))
def test_levels_of_one_sector(su2lib, kind, n):
    import torch

    from su2dmrg_gb300 import su2 as S

    rng = np.random.default_rng(n)
    u, _ = np.linalg.qr(rng.standard_normal((n, n)))
    v, _ = np.linalg.qr(rng.standard_normal((n, n)))
    s = SPECTRA[kind](np.arange(n), n)
    s = s / np.linalg.norm(s)
    a = (u * s) @ v.T
    leg = S.Su2Bond(-1, [1], [n])
    psi = S.Su2Struct([leg, leg], 0).with_legal_flags()
    half = S.Su2Struct([S.Su2Bond(1, [0], [n]), S.Su2Bond(1, [1], [1]), leg], 0)
    x = torch.from_numpy(a.ravel(order="F").copy()).cuda()
    for keep in {n, max(1, n // 2)}:
        tu, xu, _tv, xv, w = S.svd(psi, x, half, 1.0, half, 0.0, keep)
        m = tu.bonds[2].dim[0]
        U = xu.cpu().numpy()[: n * m].reshape(n, m, order="F")
        V = xv.cpu().numpy()[: n * m].reshape(n, m, order="F")
        assert np.abs(V.T @ V - np.eye(m)).max() <= 1e-13
        assert np.linalg.norm(U - a @ V) <= 1e-13
        top = np.sort(w)[::-1][: max(1, n // 2)]
        ex = np.sort(s)[::-1][: len(top)]
        assert (np.abs(top - ex) <= 1e-12 * ex[0] + 1e-15 * ex[0] ** 2 / ex).all()
        if keep == n and m == n and s.min() > 1e-7 * s.max():
            assert np.linalg.norm(U @ V.T - a) <= 1e-13
