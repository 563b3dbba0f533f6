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
extern "C" int atom_pass(double n, double ncell, double occupied) { return dpd::atom_pass(n, ncell, occupied); }
extern "C" int atom_pass_logged(double n, double occupied) { return dpd::atom_pass_logged(n, occupied); }
extern "C" int filter_pays(double half_list) { return dpd::filter_pays(half_list); }
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
    lib.atom_pass.argtypes = [ctypes.c_double] * 3
    lib.atom_pass_logged.argtypes = [ctypes.c_double] * 2
    lib.filter_pays.argtypes = [ctypes.c_double]
    lib.lists_beyond.argtypes = [ctypes.c_double, ctypes.c_double]
    return lib


def test_engines_that_share_the_gpu_take_one_warp_per_32_particles(rules):
    for warps, alone in ((1, 16), (148, 16), (149, 8), (296, 8), (297, 4), (148 * 6, 4), (148 * 6 + 1, 2),
                         (148 * 20, 2), (148 * 20 + 1, 1), (9472, 1)):
        assert rules.flat_parts(warps, 0) == 1
        assert rules.flat_parts(warps, 1) == alone


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


# us a step without thermo, measured with a warp per atom and per cell: the rule takes the faster one
# where they differ by more than a tenth
@pytest.mark.parametrize("n,rho,atom,cell", [
    (1000, 0.05, 19.0, 11.8), (1000, 0.5, 19.7, 9.6), (4000, 0.02, 20.0, 40.4), (4000, 0.05, 20.5, 27.0),
    (4000, 0.5, 21.7, 15.3), (7000, 0.1, 22.9, 33.0), (7000, 0.2, 23.3, 26.9), (7000, 0.5, 24.9, 21.2),
    (10000, 0.2, 25.9, 35.8), (10000, 1.0, 29.1, 21.6), (14000, 0.5, 29.2, 34.9), (20000, 0.5, 34.2, 47.5),
    (20000, 1.25, 39.3, 32.4), (50000, 0.75, 60.8, 84.4), (50000, 1.0, 65.1, 72.4), (50000, 1.5, 71.3, 63.5),
    (100000, 0.05, 83.3, 487.7), (100000, 1.25, 113.5, 130.3), (100000, 2.0, 123.3, 99.9), (300000, 2.0, 321.7, 293.4),
    (200000, 3.0, 2.0, 1.0), (3000000, 3.0, 2.0, 1.0),  # the densities the engine is used at: a warp per cell
])
def test_fp64_pass_is_the_faster_one(rules, n, rho, atom, cell):
    import math
    ncell = n / rho
    occupied = ncell * (1.0 - math.exp(-rho))  # atoms at random
    if abs(atom - cell) > 0.1 * min(atom, cell):
        assert bool(rules.atom_pass(n, ncell, occupied)) == (atom < cell)


def test_fp64_pass_of_atoms_that_stay_together(rules):
    # a slab of 24000 atoms at density 6 in boxes of 48000 and 96000 cells: 99 and 104 us a step with a
    # warp per cell, 109 with a warp per atom
    for ncell in (12000, 48000, 96000):
        assert not rules.atom_pass(24000, ncell, 4000)


@pytest.mark.parametrize("n,rho,by_atom", [(10000, 0.5, 1), (20000, 1.0, 1), (100000, 1.5, 1), (100000, 2.0, 0),
                                           (3000, 3.0, 0), (3000000, 3.0, 0)])
def test_fp64_pass_of_logged_steps(rules, n, rho, by_atom):
    import math
    assert rules.atom_pass_logged(n, n / rho * (1.0 - math.exp(-rho))) == by_atom


@pytest.mark.parametrize("rho,skin,pays", [(0.1, 0.3, 0), (0.3, 0.3, 0), (0.1, 1.0, 0), (0.2, 1.0, 1), (1.0, 0.3, 1),
                                           (3.0, 0.3, 1)])
def test_lists_of_dilute_systems_are_not_filtered(rules, rho, skin, pays):
    import math
    assert rules.filter_pays(rho * 2.0 / 3.0 * math.pi * (1.0 + skin) ** 3) == pays
