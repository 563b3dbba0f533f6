"""The rules that choose a step's launches (no GPU): csrc/launch_rules.h compiled with g++."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpumdpd_b200", "csrc")

WRAP = """
#include "launch_rules.h"
extern "C" int flat_parts(int warps, int alone) { return dpd::flat_parts(warps, alone != 0); }
extern "C" int lists_beyond(double list_cut, double rc) { return dpd::lists_beyond(list_cut, rc); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "wrap.cpp").write_text(WRAP)
    so = str(d / "wrap.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "wrap.cpp")], check=True)
    lib = ctypes.CDLL(so)
    lib.lists_beyond.argtypes = [ctypes.c_double, ctypes.c_double]
    return lib


def test_engines_that_share_the_gpu_take_one_warp_per_32_particles(rules):
    for warps in (1, 94, 148 * 6, 148 * 6 + 1, 148 * 20, 148 * 20 + 1, 9472):
        assert rules.flat_parts(warps, 0) == 1
        assert rules.flat_parts(warps, 1) == (4 if warps <= 148 * 6 else 2 if warps <= 148 * 20 else 1)


def test_a_list_cut_at_the_pair_cutoff_holds_nothing_beyond_it(rules):
    for k in range(50, 400):
        c = k / 100.0
        assert not rules.lists_beyond(c, c), c
        assert rules.lists_beyond(c + 0.01, c) and rules.lists_beyond(c, 0.99 * c)
