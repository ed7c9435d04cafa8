"""Kernels that start while the one before them ends: chains of applications
and solves in which every launch reads what the one before wrote, on the
default stream and on another, against the same work with a synchronisation
after every call.  Equal bit for bit: the order of every sum is fixed."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("D,nspin1,max2j", [(6, 1, 2), (40, 4, 6), (123, 5, 10), (260, 4, 12), (600, 3, 12)])
@pytest.mark.parametrize("own_stream", [False, True])
def test_chain_equals_synchronised_calls(su2lib, mode, D, nspin1, max2j, own_stream):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=nspin1, seed=D, max2j=max2j)
    psi, terms, hl, hr = w.to_device()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
    out = []
    for wait in (True, False):
        with torch.cuda.stream(stream):
            plan = HeffPlan(w.psi, terms, hl, hr, mode=mode)
            a, b = psi.clone(), torch.empty_like(psi)
            for _ in range(6):
                plan.apply(a, b)
                if wait:
                    torch.cuda.synchronize()
                a, b = b, a
                a /= a.norm()
                plan.apply(a, b)
                plan.apply(b, a)  # straight after one another
                if wait:
                    torch.cuda.synchronize()
                a /= a.norm()
            v = a.clone()
            e = [plan.lanczos(v, mlanc=5) for _ in range(3)]
        torch.cuda.synchronize()
        assert plan.status() == 0
        out.append((a.clone(), v, e))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
