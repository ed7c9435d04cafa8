"""The FP64 engine's two kinds of tiles (32 x 32, one warp per element; 8 x 8
with the contraction split over eight warps) at the sizes where they change or
go wrong: blocks smaller than a fragment and ragged ones, contractions that are
no multiple of a step or shorter than the eight warps' share, more than 32
products a block (a second window), no product at all, operands stored either
way (block Hamiltonians: transposed and not), and the sizes either side of
each threshold.

Tolerance: the sums run over at most a few thousand products of entries of one
scale, so their rounding error is below sqrt(K) 2^-53 a few times over, about
2e-14 relative (Frobenius); 1e-13 leaves the oracle the same again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,nspin1,max2j,spin0", [
    (3, 0, 1, True), (5, 1, 2, True), (9, 2, 2, False), (24, 3, 6, True), (31, 1, 4, False), (40, 40, 4, True),
    (97, 2, 12, True), (131, 7, 10, False), (200, 1, 2, True), (333, 4, 3, True), (420, 2, 12, True)])
def test_heff_matches_oracle(su2lib, oracle, D, nspin1, max2j, spin0):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=D, max2j=max2j, spin0=spin0)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=0)
    y, y2 = (torch.full_like(psi, float("nan")) for _ in range(2))
    plan.apply(psi, y)
    plan.apply(psi, y2)
    torch.cuda.synchronize()
    ref = oracle.heff_apply(oracle.HeffProblem(w.psi, w.terms, w.hl, w.hr), w.psi_data)
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-13 * np.linalg.norm(ref)
    assert torch.equal(y, y2)


def test_infinite_entries_stay_in_their_rows_and_columns(su2lib):
    """Values past a block's edge or past K never reach a stored element: one
    infinite entry of H_L (its row a) gives non-finite values only in the
    output row it feeds, exactly as the dense product."""
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=61, nspin1=0, seed=2, max2j=4)
    psi, _terms, hl, _hr = w.to_device()
    hs, hx, c = hl
    hoff, _ = hs.offsets()
    b = int(np.flatnonzero(hs.flag)[1])
    a, n = hs.block_shape(b)
    hx[int(hoff[b]) + (a - 1) + (n - 1) * a] = float("inf")  # element (a - 1, n - 1)
    plan = HeffPlan(w.psi, [], (hs, hx, c), None, mode=0)
    y = torch.empty_like(psi)
    plan.apply(psi, y)
    off, _ = w.psi.offsets()
    finite = torch.isfinite(y).cpu().numpy()
    for k in np.flatnonzero(w.psi.flag):
        m, d = w.psi.block_shape(int(k))
        blk = finite[int(off[k]): int(off[k]) + m * d].reshape(m, d, order="F")
        if w.psi.block_angm(int(k))[0] == hs.block_angm(b)[0]:
            assert blk[: n - 1].all() and not blk[n - 1].any()
        else:
            assert blk.all()
