"""A cluster's CTAs write into one another's shared memory, which they may do
only once all of them are known to run: every kernel that sums over a cluster
arrives at the cluster's barrier before it waits for its predecessor, and waits
at that barrier before its first sum.  The order is read from the source (a CTA
that starts late cannot be brought about); on the GPU, solves whose vectors go
through one cluster run while another stream keeps the SMs busy, so that the
CTAs start at different times, and give the bits of a quiet GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "su2dmrg_gb300", "csrc")


def _kernels(text):
    """(name, body) of every __global__ function defined in text."""
    for m in re.finditer(r"__global__\s+void[^;{]*?(\w+)\s*\([^{};]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end(): i]


def test_cluster_kernels_wait_for_all_their_ctas():
    seen = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for kernel, body in _kernels(text):
            if "cluster_sum(" not in body:
                continue
            seen.append(kernel)
            assert body.count("cluster_arrive();") == 1 and body.count("cluster_wait();") == 1, kernel
            assert body.index("cluster_arrive();") < body.index("wait_for_predecessor()"), kernel
            assert body.index("cluster_arrive();") < body.index("cluster_wait();") < body.index("cluster_sum("), kernel
    assert len(seen) == 4, seen


@pytest.mark.gpu
@pytest.mark.parametrize("D", [3, 45, 64, 90, 128])  # 1, 1, 2, 4 and 8 elements a thread
def test_solves_beside_a_busy_stream(su2lib, D):
    import torch

    from su2dmrg_gb300.su2 import HeffPlan
    from su2dmrg_gb300.workloads import synthetic_heff

    w = synthetic_heff(D=D, nspin1=0, seed=D, max2j=0)
    psi, terms, hl, hr = w.to_device()
    plan = HeffPlan(w.psi, terms, hl, hr, mode=0)
    quiet = psi.clone()
    ref = plan.lanczos(quiet, mlanc=5)
    big = torch.randn(1 << 22, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(side):
            for _ in range(40):
                big.mul_(1.0)
        v = psi.clone()
        assert plan.lanczos(v, mlanc=5) == ref
        assert torch.equal(v, quiet)
    torch.cuda.synchronize()
