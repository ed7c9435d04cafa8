"""The rule by which a refinement level of the truncation takes a correction
step or goes to the eigensolver (csrc/svd_levels.hpp, compiled for the host): a
level that leaves a subspace beyond the cut is the last one, its values are
reported as they are, so it needs the eigensolver after whichever step shows it;
and the rules that hold for every step."""
import ctypes
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "svd_levels.hpp"
extern "C" int settled(const double* h, int n, double step, int it, double cut) {
  return su2g::level_settled(std::vector<double>(h, h + n), step, it, cut);
}
"""


@pytest.fixture(scope="module")
def settled(tmp_path_factory):
    d = tmp_path_factory.mktemp("levels")
    (d / "shim.cpp").write_text(SHIM)
    out = str(d / "levels.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I",
                    os.path.join(REPO, "su2dmrg_gb300", "csrc"), str(d / "shim.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.settled.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_int, ctypes.c_double]

    def call(h, step=1e-9, it=0, cut=0.0):
        a = (ctypes.c_double * len(h))(*h)
        return bool(lib.settled(ctypes.addressof(a), len(h), step, it, cut))

    return call


LEVEL = [3e-5, 1e-5, 2e-5, 0.11, 0.5, 1.0]  # unsorted below its decade, as a step leaves it


@pytest.mark.parametrize("it", [0, 1, 2, 3])
def test_the_last_level_before_the_cut_goes_to_the_eigensolver(settled, it):
    assert settled(LEVEL, it=it)                   # nothing is cut
    assert settled(LEVEL, it=it, cut=1.9e-4)       # 2e-5 may still hold kept values
    assert not settled(LEVEL, it=it, cut=2.1e-4)   # it does not: no further level
    assert settled([2e-5, 0.2, 1.0], it=it, cut=1.0)  # one value left: no subspace


@pytest.mark.parametrize("it", [0, 1])
def test_rules_of_every_step(settled, it):
    assert settled(LEVEL, step=9e-4, it=it)
    assert settled(LEVEL, step=9e-3, it=it) == (it > 0)
    assert not settled(LEVEL, step=2e-2, it=it)
    assert not settled([1e-5, 0.5, 0.11, 1.0], it=it)     # the decade out of order
    assert not settled([0.11, 1e-5, 0.5, 1.0], it=it)     # one of the decade below the rest
    assert not settled([-3e-17, -1e-17], it=it)           # no positive value
