"""The rules that divide an update's work (csrc/sph_rules.h), on the CPU."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "sph_rules.h"
using namespace sphgb;
extern "C" {
int halves(int cells, int live, int added, int sms) { return density_halves(cells, live, added, sms); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "nbodysimulation_experiment_gb300", "csrc"), str(d / "shim.cpp"), "-o", so])
    return ctypes.CDLL(so)


@pytest.mark.parametrize("cells, live, added, want", [
    (1590, 114, 0, 1),        # the 4,096-particle dam break in its box
    (262144, 120, 0, 1),      # a small scene in a large box
    (2400, 2400, 0, 1),
    (16500, 16500, 0, 0),     # a full box
    (3000, 3000, 0, 0),
    (4864, 4800, 0, 0),
    (6000, 6000, 0, 1),       # a last wave nearly empty with one warp a cell
    (65280, 6000, 0, 0),
    (1048576, 120, 0, 0),     # mostly empty cells to pass over
    (1590, 0, 4096, 1),       # the same scenes' first updates
    (16500, 0, 594000, 0),
])
def test_density_halves(rules, cells, live, added, want):
    assert rules.halves(cells, live, added, 152) == want
