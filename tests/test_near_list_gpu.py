"""Many-body DPD where the density pass's queue and near list can go wrong: particles with more
entries inside rd than a column of the queue holds, none at all, cutoffs below the list's, the
density and the forces against the oracle."""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("rho,vapour,skin", [(6.0, 0.0, 0.3), (25.0, 0.05, 0.3), (40.0, 0.0, 0.0), (1.0, 0.3, 0.5)])
def test_density_and_forces_match_oracle(oracle_mod, mode, rho, vapour, skin):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.mdpd_slab(Lx=5.5, Ly=5.5, Lz=14.0, z0=4.0, z1=9.0, rho=rho, rho_vapour=vapour, seed=91, dt=0.001,
                         skin=skin, nsteps=3, max_rho=120.0)
    e = Engine(s.run_in, system=s.c_system())
    e.set_tuning(launch_mode=mode)
    for n in (0, 2):
        e.run(n)
        st, c = e.state(), e.cells()
        L = c["nc"].astype(np.float64) * c["w"].astype(np.float64)
        ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
        if n == 0:  # forces of the state's own positions and velocities
            o = oracle_mod.forces(ff, np.arange(1, s.n + 1), s.types, st["x"], st["v"], s.lo, L, 0)
            assert force_err(st["f"], o["f"]) < 1e-5
            np.testing.assert_allclose(e.density(), o["rho"], rtol=1e-5, atol=1e-5 * max(rho, 1.0))
    e.close()
