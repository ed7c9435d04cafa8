"""All slots' layouts in one call (su2g_env_layouts) against one call per slot,
and batches whose jobs share operator structures against batches of one job:
operators of one structure, of different stored blocks, of different spins,
repeated slots, both sides."""

import numpy as np
import pytest


def _jobs(S, w, rng, mixed):
    jobs = []
    for i, (s, x) in enumerate(w.ops):
        if mixed and i % 2:
            t = S.Su2Struct(list(s.bonds), 0)
            keep = rng.random(len(s.flag)) < 0.7
            t.flag = (s.flag * keep).astype(np.int32)
            if not t.flag.any():
                t.flag = s.flag.copy()
            s = t
        jobs.append({"kind": "transform", "slot": i, "coef": 1.0 + i, "x": (s, x)})
    n = len(w.ops)
    jobs.append({"kind": "overlap", "slot": n, "x": (w.hh[0], w.hh[1])})
    jobs.append({"kind": "transform", "slot": 0, "coef": -0.5, "x": jobs[1]["x"]})
    jobs.append({"kind": "overlap", "slot": n, "coef": 2.0, "x": (w.hh[0], w.hh[1])})
    return jobs, n + 1


@pytest.mark.parametrize("D,nops,max2j", [(8, 2, 2), (40, 3, 6), (150, 5, 12)])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("flag", [0, 1])
def test_all_slots_at_once(su2lib, D, nops, max2j, mixed, flag):
    from su2dmrg_gb300 import capi
    from su2dmrg_gb300 import su2 as S
    from su2dmrg_gb300.workloads import synthetic_site_step

    w = synthetic_site_step(D=D, nops=nops, seed=7, max2j=max2j)
    su, du = w.uu
    if flag:
        su = S.Su2Struct([su.bonds[1], su.bonds[0], su.bonds[2]], 0).with_legal_flags()
    jobs, n = _jobs(S, w, np.random.default_rng(D), mixed)
    keep = []
    J = S._EnvJobs(jobs)
    tu = S._tensor(su, du, keep)
    stride = 4 + 3 * (2 + 2 * 64)
    desc, flags, size = np.zeros((n, stride), np.int32), np.zeros(n * 64 ** 2, np.int32), np.zeros(n, np.int64)
    capi.check(capi.lib().su2g_env_layouts(tu, tu, flag, J.n, J.ptr, n, S.ptr(desc), stride, S.ptr(flags), len(flags),
                                           S.ptr(size)))
    at = 0
    for s in range(n):
        one = S.env_layout(su, du, su, du, flag, jobs, s)
        got = S._parse_desc(desc[s])
        assert got.desc().tolist() == one.desc().tolist()
        assert flags[at: at + got.nten].tolist() == one.flag.tolist()
        assert size[s] == one.size()
        at += got.nten


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("D,max2j", [(8, 2), (60, 8)])
def test_shared_structures_plan_like_single_jobs(su2lib, mode, D, max2j):
    """The products of a batch are those of its jobs, one by one."""
    from su2dmrg_gb300 import su2 as S
    from su2dmrg_gb300.workloads import synthetic_site_step

    w = synthetic_site_step(D=D, nops=3, seed=11, max2j=max2j)
    su, du = w.uu
    jobs, n = _jobs(S, w, np.random.default_rng(5), True)
    whole = S.env_validate(su, du, su, du, 0, jobs, mode=mode)["flops"]
    alone = sum(S.env_validate(su, du, su, du, 0, [dict(j, slot=0)], mode=mode)["flops"] for j in jobs)
    assert whole == alone


def test_too_small_arrays_are_refused(su2lib):
    from su2dmrg_gb300 import capi
    from su2dmrg_gb300 import su2 as S
    from su2dmrg_gb300.workloads import synthetic_site_step

    w = synthetic_site_step(D=20, nops=2, seed=1, max2j=4)
    su, du = w.uu
    jobs, n = _jobs(S, w, np.random.default_rng(1), False)
    keep, J = [], S._EnvJobs(jobs)
    tu = S._tensor(su, du, keep)
    desc, flags, size = np.zeros((n, 400), np.int32), np.zeros(64, np.int32), np.zeros(n, np.int64)
    rc = capi.lib().su2g_env_layouts(tu, tu, 0, J.n, J.ptr, n, S.ptr(desc), 400, S.ptr(flags), 3, S.ptr(size))
    assert rc == capi.SU2G_EINVAL
    rc = capi.lib().su2g_env_layouts(tu, tu, 0, J.n, J.ptr, n, S.ptr(desc), 2, S.ptr(flags), 64, S.ptr(size))
    assert rc == capi.SU2G_EINVAL
