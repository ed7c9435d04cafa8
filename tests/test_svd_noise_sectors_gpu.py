"""Several sectors of a truncation whose matrices are known to their rounding
only (rank well below their size, as a warm-up's are until the bond dimension
binds): their last refinement levels have negative eigenvalues larger than any
positive one, and the sectors' decompositions go through the eigensolver
together, padded to one size.

Whatever the noise, the new V's columns are orthonormal (1e-13, as in the other
tests of the levels: a chain of orthogonal rotations), U = psi V, the values
are the columns' norms where they lie above the noise (the Gram method's bound
1e-15 s_max^2 / s + 1e-12 s_max), and psi = U V^T to 1e-7 s_max: what the
dropped directions (negative eigenvalues, in magnitude below a few n 2^-53
s_max^2) can hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rank", [([2, 1, 3], 1), ([9, 4, 17, 2], 2), ([27, 53, 46, 31, 18, 8, 1], 12),
                                       ([60, 128, 129, 7, 33], 20), ([64, 64, 64], 40), ([90, 30, 140, 110], 5)])
@pytest.mark.parametrize("graded", [False, True])
def test_low_rank_sectors(su2lib, dims, rank, graded):
    import torch

    from su2dmrg_gb300 import su2 as S

    rng = np.random.default_rng(sum(dims) + rank)
    ang = list(range(len(dims)))
    leg = S.Su2Bond(-1, ang, dims)
    psi = S.Su2Struct([leg, leg], 0).with_legal_flags()
    tu = S.Su2Struct([S.Su2Bond(1, ang, dims), S.Su2Bond(1, [0], [1]), leg], 0)
    off, total = psi.offsets()
    x = np.zeros(total)
    mats = {}
    for b in np.flatnonzero(psi.flag):
        n = psi.block_shape(int(b))[0]
        r = min(rank, n)
        s = np.exp(-(20.0 if graded else 2.0) * np.arange(r) / max(r, 1))
        a = (rng.standard_normal((n, r)) * s) @ rng.standard_normal((r, n)) / n
        mats[psi.block_angm(int(b))[0]] = a
        x[off[b]: off[b] + n * n] = a.ravel(order="F")
    norm = np.linalg.norm(x)
    ts, xu, vs, xv, w = S.svd(psi, torch.from_numpy(x / norm).cuda(), tu, 1.0, tu, 0.0, sum(dims))
    uoff, _ = ts.offsets()
    xu, xv = xu.cpu().numpy(), xv.cpu().numpy()
    seen = 0
    for b in np.flatnonzero(ts.flag):
        j = ts.block_angm(int(b))[2]
        n, _, m = ts.block_shape(int(b))
        a = mats[j] / norm
        U = xu[uoff[b]: uoff[b] + n * m].reshape(n, m, order="F")
        V = xv[uoff[b]: uoff[b] + n * m].reshape(n, m, order="F")
        assert np.abs(V.T @ V - np.eye(m)).max() <= 1e-13
        assert np.abs(U - a @ V).max() <= 1e-13
        top = np.linalg.svd(a, compute_uv=False)
        assert np.linalg.norm(U @ V.T - a) <= 1e-7 * top[0]
        s = np.sort(np.linalg.norm(U, axis=0))[::-1]
        k = min(m, int((top > 1e-6 * top[0]).sum()))
        assert (np.abs(s[:k] - top[:k]) <= 1e-12 * top[0] + 1e-15 * top[0] ** 2 / top[:k]).all()
        seen += m
    assert seen == len(w)
