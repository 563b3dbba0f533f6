"""Many-body DPD over steps that reuse the neighbour list: the density pass then filters the list of
an earlier step by the present positions, and what it leaves must be all pairs inside the cutoff.

After every few steps the density and the forces are compared with the oracle's at the state's own
positions and at the velocities the step's forces were taken with (the state's, less the final half
kick), to the tolerance of the step-0 tests.
"""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("rho,vapour,skin,dt", [(6.0, 0.0, 0.3, 5e-4), (25.0, 0.05, 0.3, 1e-4), (1.0, 0.3, 0.5, 5e-4)])
def test_reused_list_gives_the_oracle_density_and_forces(oracle_mod, mode, rho, vapour, skin, dt):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.mdpd_slab(Lx=5.5, Ly=5.5, Lz=14.0, z0=4.0, z1=9.0, rho=rho, rho_vapour=vapour, seed=91, dt=dt,
                         skin=skin, nsteps=30, max_rho=120.0)
    e = Engine(s.run_in, system=s.c_system())
    e.set_tuning(launch_mode=mode)
    c = e.cells()
    box = c["nc"].astype(np.float64) * c["w"].astype(np.float64)
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    e.run(0)
    x0, reused = e.state()["x"], 0
    for _ in range(4):
        builds = e.info()["builds"]
        e.run(5)
        reused += e.info()["builds"] == builds
        st = e.state()
        o = oracle_mod.forces(ff, np.arange(1, s.n + 1), s.types, st["x"], st["v"] - 0.5 * dt * st["f"], s.lo, box,
                              e.info()["step"])
        assert force_err(st["f"], o["f"]) < 1e-5
        np.testing.assert_allclose(e.density(), o["rho"], rtol=1e-5, atol=1e-5 * max(rho, 1.0))
    drift = st["x"] - x0
    drift -= box * np.round(drift / box)
    assert reused >= 2 and np.abs(drift).max() > 5e-3
    e.close()
