"""The FP64 engine's steps without thermo, whose force pass also takes the atoms to the next step and
into their next cells: positions, velocities, forces, image counters and thermo rows against the FP64
oracle, in runs cut so that such steps and separate ones (logged steps, the last of a run) alternate.

Tolerances are those of the engine's other oracle tests: only FP64 summation order separates the two.
"""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


def _system(name, thermo):
    from gpumdpd_b200 import inputs
    k = dict(seed=93, dt=0.02, nsteps=10, thermo=thermo, skin=0.0, max_rho=40.0)
    if name == "boxes_of_3_cells":
        return inputs.plain_dpd(L=3.0, rho=3.0, **k)
    if name == "dense_cells":  # more atoms in a cell than a round takes, more neighbours than are staged
        return inputs.plain_dpd(L=3.2, rho=13.0, **dict(k, dt=0.005))
    if name == "empty_cells":
        return inputs.plain_dpd(L=9.0, rho=0.4, **k)
    if name == "many_body":
        return inputs.mdpd_slab(Lx=4.5, Ly=4.5, Lz=9.0, z0=2.0, z1=7.0, rho=6.0, rho_vapour=0.2, **dict(k, dt=0.01))
    if name == "bonds":
        return inputs.diblock_melt(L=5.5, **k)
    if name == "angles":
        return inputs.angle_chains(L=5.5, **k)
    s = inputs.binary_mixture(L=5.2, a_ab=40.0, **{q: k[q] for q in k})
    if name == "half_integrated":  # type 2 stays where it is
        s.run_in = s.run_in.replace("group all type 1 2", "group a type 1").replace("fix md all nve", "fix md a nve")
        assert "fix md a nve" in s.run_in and "group a type 1\n" in s.run_in
    return s


@pytest.mark.parametrize("thermo", [100, 3])
@pytest.mark.parametrize("name", ["boxes_of_3_cells", "dense_cells", "empty_cells", "many_body", "bonds", "angles",
                                  "mixture", "half_integrated"])
def test_steps_without_thermo_match_oracle(oracle_mod, name, thermo):
    from gpumdpd_b200 import Engine
    s = _system(name, thermo)
    e = Engine(s.run_in, system=s.c_system(), precision="fp64")
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    box = s.hi - s.lo
    done, moved = 0, 0
    for n in (3, 1, 4):
        e.run(n)
        done += n
        st = e.state()
        oracle_mod.set_saru_double_tail(True)
        try:
            o = oracle_mod.run(ff, np.arange(1, s.n + 1), s.types, s.x, s.v, s.lo, box, 1, done, thermo,
                               bonds=s.bonds, angles=getattr(s, "angles", None))
        finally:
            oracle_mod.set_saru_double_tail(False)
        dx = (st["x"] + st["image"] * box) - (o["x"] + o["image"] * box)  # unwrapped: images count
        assert np.abs(dx).max() < 1e-9
        assert np.abs(st["v"] - o["v"]).max() < 1e-9
        assert force_err(st["f"], o["f"]) < 1e-9
        assert (st["x"] >= s.lo).all() and (st["x"] < s.hi).all()
        moved = int(np.abs(o["image"]).sum())
    assert moved > 0  # some atom has crossed the boundary
    th = e.thermo()
    assert list(th["step"]) == [k for k in range(done + 1) if k % thermo == 0]
    for k in ("temp", "pair_pe", "bond_pe", "angle_pe", "pressure"):
        np.testing.assert_allclose(th[k], o["thermo"][k], rtol=1e-9, atol=1e-9)
    e.close()
