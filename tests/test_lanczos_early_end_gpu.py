"""A long solve whose recurrence ends at its second step does no more
applications than it reports: the two steps and the eigenvector's check, three
applications in all.  H_L = diag(+-1) has two eigenvalues, so the second norm
vanishes.  Five applications would run if the host looked at the coefficients
only at the fourth step; a solve of three takes little more than three
(some dozen passes over vectors of 1.4 and 25 million elements),
so anything below four says that the late steps did not run."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,D", [(0, 1200), (1, 5000)])
def test_no_steps_after_the_end(su2lib, mode, D):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=0, seed=1, max2j=0)
    h = torch.diag(torch.where(torch.arange(D) % 2 == 0, -1.0, 1.0).double()).cuda().ravel().contiguous()
    plan = HeffPlan(w.psi, [], (w.hl[0], h, 1.0), None, mode=mode)
    x = torch.from_numpy(w.psi_data).cuda()
    y = torch.empty_like(x)

    def best(f):
        took = []
        for _ in range(8):
            torch.cuda.synchronize()
            t = time.perf_counter()
            f()
            torch.cuda.synchronize()
            took.append(time.perf_counter() - t)
        return min(took)

    energy, matvecs = plan.lanczos(x.clone(), mlanc=5)
    assert matvecs == 3 and abs(energy + 1.0) <= 1e-12
    one = best(lambda: plan.apply(x, y))
    solve = best(lambda: plan.lanczos(x.clone(), mlanc=5))
    print(f"mode {mode}, D = {D}: application {one * 1e3:.3f} ms, solve {solve * 1e3:.3f} ms")
    assert solve < 4 * one
    assert plan.status() == 0
