"""The FP64 launch lists of a phase with tiles in plenty: a site update of many
operators, launched as the planner cuts it (under any tile table) or cut but
not sorted, against the same update a few operators at a time.  Equal bit for
bit: whole tiles of any shape sum an element's products in the same order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nops", [30, 180])  # phase 1: 46 and 274 tiles of 32 x 32 an SM, 10 in the small batch
def test_many_operators_equal_a_few_at_a_time(su2lib, nops):
    import torch

    from su2dmrg_gb300 import autotune as A
    from su2dmrg_gb300 import su2 as S
    from su2dmrg_gb300.workloads import synthetic_site_step

    w = synthetic_site_step(D=700, nops=6)
    su, xu = w.uu
    du = torch.from_numpy(xu).cuda()
    ops = [(s, torch.from_numpy(x).cuda()) for s, x in w.ops]
    torch.cuda.synchronize()
    jobs = [{"kind": "transform", "slot": t, "x": ops[t % 6]} for t in range(nops)]
    few = [y.clone() for _, y in S.env_batch(su, du, su, du, 0, jobs[:6])]
    try:
        for cls in (0, 1, 2, 3, None):
            A.load() if cls is None else A.install({"m_edges": [], "n_edges": [], "cls": [cls]})
            many = S.env_batch(su, du, su, du, 0, jobs)
            torch.cuda.synchronize()
            for t, (_, y) in enumerate(many):
                assert torch.equal(y, few[t % 6])
    finally:
        A.load()
