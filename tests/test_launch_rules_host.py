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
extern "C" int pair_schedule(int asked, int tile, int small, int entry)
{
    return dpd::pair_schedule(asked, tile != 0, small != 0, entry != 0);
}
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


def test_names_of_one_schedule_are_launched_alike(rules):
    for tile, small, entry in ((0, 0, 0), (0, 1, 0), (0, 1, 1)):
        want = rules.pair_schedule(8, tile, small, entry)
        assert want == (10 if entry else 4 if small else 8)
        for other in (7, 9, 11):  # 11: an engine without the cell tiles
            assert rules.pair_schedule(other, tile, small, entry) == want
        for own in (0, 1, 2, 3, 4, 5, 6, 10):
            assert rules.pair_schedule(own, tile, small, entry) == own
    assert rules.pair_schedule(11, 1, 1, 0) == 11


def test_the_tuner_times_a_schedule_once(rules):
    from gpumdpd_b200 import tune
    names = [(rules.pair_schedule(s["pair_variant"], s["pair_variant"] == 11, 0, 0), s.get("tile")) for s in tune.SCHEDULES]
    assert len(set(names)) == len(names)
