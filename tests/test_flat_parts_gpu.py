"""The flattened pair schedule with 32 particles shared by 16, 8 and 4 warps: step-0 forces and thermo
against the oracle at the sizes where the split changes, on lists longer than a round of the filter
takes, lists with fewer entries than parts, and with bonds and many-body forces."""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


def _system(kind, n, skin):
    from gpumdpd_b200 import inputs
    k = dict(seed=95, dt=0.005, nsteps=10, thermo=1, skin=skin)
    if kind == "sparse":  # a few entries a particle or none
        return inputs.plain_dpd(L=(n / 0.5) ** (1 / 3), rho=0.5, **k)
    if kind == "dense":
        return inputs.plain_dpd(L=(n / 16.0) ** (1 / 3), rho=16.0, max_rho=40.0, **k)
    if kind == "chains":
        return inputs.diblock_melt(L=(n / 3.0) ** (1 / 3), **k)
    L = (n / 6.0 * 3.0) ** (1 / 3)  # the liquid in a third of the box
    return inputs.mdpd_slab(Lx=L, Ly=L, Lz=L, z0=L / 3, z1=2 * L / 3, rho=6.0, max_rho=40.0, **k)


@pytest.mark.parametrize("skin", [0.0, 0.3])
@pytest.mark.parametrize("n", [1100, 4700, 4800, 9400, 9550])  # 148 and 296 warps lie between
@pytest.mark.parametrize("kind", ["sparse", "dense", "chains", "many_body"])
def test_forces_of_shared_particles(oracle_mod, kind, n, skin):
    from gpumdpd_b200 import Engine
    s = _system(kind, n, skin)
    e = Engine(s.run_in, system=s.c_system())
    e.set_tuning(pair_variant=4)
    e.run(0)
    st, c = e.state(), e.cells()
    L = c["nc"].astype(np.float64) * c["w"].astype(np.float64)
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    o = oracle_mod.forces(ff, np.arange(1, s.n + 1), s.types, st["x"], st["v"], s.lo, L, 0, bonds=s.bonds)
    assert force_err(st["f"], o["f"]) < 1e-5
    th = e.thermo()
    assert th["pair_pe"][0] == pytest.approx(o["pair_pe"], rel=1e-5)
    assert th["bond_pe"][0] == pytest.approx(o["bond_pe"], rel=1e-5, abs=1e-9)
    e.close()
