"""Large grids with a skin: dilute systems, whose lists the flattened pair pass takes unfiltered, and
drops in an otherwise empty box, whose lists it filters.  Forces of a fresh list and of a list of
earlier steps, and the thermo row, against the oracle."""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


def _system(kind):
    from gpumdpd_b200 import inputs
    k = dict(seed=96, dt=0.002, nsteps=10, thermo=1, skin=0.3)
    if kind == "gas":
        return inputs.plain_dpd(L=101.0, rho=0.3, **k)  # 309090 particles: 1208 blocks of 256 slots
    if kind == "chains":
        return inputs.diblock_melt(L=101.0, rho=0.3, **k)
    s = inputs.plain_dpd(L=150.0, rho=0.0915, max_rho=25.0, **dict(k, dt=0.0005))  # "drop"
    x = np.random.default_rng(3).uniform(0.0, 46.0, (s.n, 3))
    return inputs.System(s.lo, s.hi, s.masses, s.types, x, s.v, run_in=s.run_in)


@pytest.mark.parametrize("kind", ["gas", "chains", "drop"])
def test_forces_on_fresh_and_reused_lists(oracle_mod, kind):
    from gpumdpd_b200 import Engine
    s = _system(kind)
    dt = 0.0005 if kind == "drop" else 0.002
    e = Engine(s.run_in, system=s.c_system())
    c = e.cells()
    box = c["nc"].astype(np.float64) * c["w"].astype(np.float64)
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    for n in (0, 4):
        e.run(n)
        st = e.state()
        v = st["v"] - (0.5 * dt * st["f"] if n else 0.0)  # the velocities of the force evaluation
        o = oracle_mod.forces(ff, np.arange(1, s.n + 1), s.types, st["x"], v, s.lo, box, e.info()["step"], bonds=s.bonds)
        assert force_err(st["f"], o["f"]) < 1e-5
        th = e.thermo(1)
        assert th["pair_pe"][0] == pytest.approx(o["pair_pe"], rel=1e-5)
        assert th["bond_pe"][0] == pytest.approx(o["bond_pe"], rel=1e-5, abs=1e-9)
    assert e.info()["builds"] == 1
    e.close()
