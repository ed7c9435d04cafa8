"""The FP64 launch lists (f64_launch_tiles) of phases with many output blocks:
a site update of a large run, whose tiles would be cut into hundreds of
thousands of 8 x 8 ones by the length of their contraction alone, at a host
cost of several device times.  From the structures alone, compiled for the host
with the planners: what is launched never outnumbers the 32 x 32 tiles once an
SM gets 64 of them or more, covers exactly the planner's tiles, sums the same
way under every tile table, and short phases are still split."""
import ctypes
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "su2dmrg_gb300", "csrc")
ADDR = 1 << 40  # operands are never read: planning only needs addresses

SHIM = r"""
#include "env_plan.hpp"
using namespace su2g;
namespace {
void count(const std::vector<GemmTile>& planned, int64_t* r) {
  for (int i = 0; i < 5; ++i) r[i] = 0;
  r[0] = (int64_t)planned.size();
  int64_t area = 0;
  for (const GemmTile& t : planned) {
    r[1] += (int64_t)((t.mlen + 31) / 32) * ((t.nlen + 31) / 32);
    area += (int64_t)t.mlen * t.nlen * (t.c % 1009 + t.seg0 + 1);
  }
  const std::vector<GemmTile> out = f64_launch_tiles(planned);
  r[2] = (int64_t)out.size();
  for (const GemmTile& t : out) {
    r[3] += t.ksplit;
    area -= (int64_t)t.mlen * t.nlen * (t.c % 1009 + t.seg0 + 1);
  }
  r[4] = area;
}
}  // namespace
extern "C" int one_class(int cls) {
  const int open = 1 << 30;
  return set_tile_table(&open, 1, &open, 1, &cls);
}
extern "C" int env_lists(su2g_tensor u, int nj, const su2g_env_job* jobs, int nslots, double* const* outs, int64_t* r) {
  HeffWork w;
  std::vector<Struct> ys;
  std::string err;
  const int rc = build_env_batch(u, u, 0, nj, jobs, nslots, outs, &w, &ys, &err);
  if (rc) return rc;
  count(w.tile1, r);
  count(w.tile2, r + 5);
  return 0;
}
extern "C" int heff_lists(const int* d, const int* f, int nt, const su2g_term* t, const su2g_tensor* h, int64_t* r) {
  HeffWork w;
  std::string err;
  const int rc = build_heff_work(d, f, nt, t, h, 1.0, h, 1.0, &w, &err);
  if (rc) return rc;
  count(w.tile1, r);
  count(w.tile2, r + 5);
  return 0;
}
extern "C" int input_lists(su2g_tensor l, su2g_tensor r_, int64_t* r) {
  HeffWork w;
  Struct v;
  std::string err;
  double* at = reinterpret_cast<double*>((uintptr_t)1 << 40);
  const int rc = build_input_vector(l, r_, at, at, &v, &w, &err);
  if (rc) return rc;
  count(w.tile1, r);
  count(w.tile2, r + 5);
  return 0;
}
"""


class _Device:
    """An operand that stands for device memory."""

    is_cuda = True

    def data_ptr(self):
        return ADDR


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    from su2dmrg_gb300 import capi

    d = tmp_path_factory.mktemp("lists")
    (d / "shim.cpp").write_text(SHIM)
    out = str(d / "lists.so")
    srcs = [str(d / "shim.cpp")] + [os.path.join(CSRC, s) for s in ("heff_plan.cpp", "env_plan.cpp", "su2_meta.cpp")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", CSRC,
                    "-I", os.path.join(REPO, "include"), *srcs, "-o", out], check=True)
    lib = ctypes.CDLL(out)
    i, p = ctypes.c_int, ctypes.c_void_p
    lib.env_lists.argtypes = [capi.Tensor, i, p, i, p, p]
    lib.heff_lists.argtypes = [p, p, i, p, p, p]
    lib.input_lists.argtypes = [capi.Tensor, capi.Tensor, p]
    return lib


def _bond(D, direction, max2j=12):
    from su2dmrg_gb300.su2 import Su2Bond
    from su2dmrg_gb300.workloads import gaussian_sector_counts

    c = gaussian_sector_counts(D, max2j)
    a = [k for k in range(max2j + 1) if c[k]]
    return Su2Bond(direction, a, [c[k] for k in a])


def _lists(planner, kind, D, n):
    """[(planned, 32 x 32 tiles, launched, split ones, area missing)] of both phases."""
    from su2dmrg_gb300 import su2 as S

    r = (ctypes.c_int64 * 10)()
    half, x, keep = S.Su2Bond(1, [1], [1]), _Device(), []
    if kind == "env":
        u = S.Su2Struct([_bond(D, -1), half, _bond(D, 1)], 0).with_legal_flags()
        op = S.Su2Struct([_bond(D, 1), S.Su2Bond(-1, [2], [1]), _bond(D, -1)], 0).with_legal_flags()
        h = S.Su2Struct([_bond(D, 1), _bond(D, -1)], 0).with_legal_flags()
        jobs = [{"kind": "transform", "slot": t, "x": (op, x)} for t in range(n)]
        J = S._EnvJobs(jobs + [{"kind": "overlap", "slot": n, "x": (h, x)}])
        outs = (ctypes.c_void_p * (n + 1))(*[ADDR] * (n + 1))
        rc = planner.env_lists(S._tensor(u, x, keep), J.n, J.ptr, n + 1, ctypes.addressof(outs), ctypes.addressof(r))
    elif kind == "heff":
        enl = _bond(D, 1).fuse(half)
        enl.dir = -1
        inb = enl.inverted()
        st = S.Su2Struct([enl, enl], 0).with_legal_flags()
        psi = S._Pinned(st)
        op = S.Su2Struct([inb, S.Su2Bond(1, [2], [1]), enl], 0).with_legal_flags()
        h = S._tensor(S.Su2Struct([inb, enl], 0).with_legal_flags(), x, keep)
        a = S._PlanArgs(st, [(op, x, op, x, 1.0)] * n, None, None)
        rc = planner.heff_lists(psi.pdesc, psi.pflag, n, ctypes.addressof(a.tarr), ctypes.addressof(h),
                                ctypes.addressof(r))
    else:
        ul = S.Su2Struct([_bond(D, 1), half, _bond(D, -1)], 0).with_legal_flags()
        ur = S.Su2Struct([half, _bond(D, 1), _bond(D, -1)], 0).with_legal_flags()
        rc = planner.input_lists(S._tensor(ul, x, keep), S._tensor(ur, x, keep), ctypes.addressof(r))
    assert rc == 0
    return [tuple(r[5 * k: 5 * k + 5]) for k in (0, 1)]


@pytest.mark.parametrize("kind,D,n", [
    ("env", 700, 18), ("env", 1500, 18), ("env", 1900, 3), ("env", 2000, 4), ("env", 2000, 18), ("env", 4000, 18),
    ("heff", 700, 12), ("heff", 2000, 18), ("heff", 4000, 18), ("input", 2000, 0), ("input", 8000, 0)])
def test_lists_stay_short_where_tiles_are_plenty(planner, kind, D, n):
    for cls in (0, 3):
        assert planner.one_class(cls) == 0
        for planned, whole, launched, split, missing in _lists(planner, kind, D, n):
            assert missing == 0
            if whole >= 64 * 152:
                assert launched <= whole and split == 0
            assert launched <= max(whole, 128 * 1024)  # 8 MB, whatever the phase


@pytest.mark.parametrize("kind,D,n", [("env", 150, 6), ("env", 2000, 18), ("heff", 123, 5), ("heff", 2000, 18)])
def test_the_table_does_not_decide_how_a_phase_sums(planner, kind, D, n):
    got = []
    for cls in range(4):
        assert planner.one_class(cls) == 0
        got.append([split > 0 for _, _, _, split, _ in _lists(planner, kind, D, n)])
    assert all(g == got[0] for g in got)


@pytest.mark.parametrize("D,n", [(24, 2), (123, 5), (251, 9), (1000, 18), (2000, 18)])
def test_few_long_contractions_are_split(planner, D, n):
    assert planner.one_class(0) == 0
    assert _lists(planner, "heff", D, n)[1][3] > 0
