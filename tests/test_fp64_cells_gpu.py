"""The FP64 engine's force pass by cells where its rounds and images can go wrong: boxes of 3
cells (every neighbouring cell across the boundary), cells of more atoms than a round takes,
neighbourhoods larger than the staged records, sparse boxes with empty cells."""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,rho", [(3.0, 3.0), (3.2, 13.0), (4.7, 6.0), (9.0, 0.4)])
def test_cell_rounds_and_images_match_oracle(oracle_mod, L, rho):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.plain_dpd(L=L, rho=rho, seed=91, dt=0.005, nsteps=10, thermo=1, max_rho=40.0, skin=0.0)
    e = Engine(s.run_in, system=s.c_system(), precision="fp64")
    e.run(4)
    st = e.state()
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    box = s.hi - s.lo
    oracle_mod.set_saru_double_tail(True)
    try:
        o = oracle_mod.run(ff, np.arange(1, s.n + 1), s.types, s.x, s.v, s.lo, box, 1, 4, 1)
    finally:
        oracle_mod.set_saru_double_tail(False)
    dx = st["x"] - o["x"]
    dx -= box * np.round(dx / box)
    # FP64 summation order, as the engine's other oracle tests
    assert np.abs(dx).max() < 1e-9
    assert np.abs(st["v"] - o["v"]).max() < 1e-9
    assert force_err(st["f"], o["f"]) < 1e-9
    th = e.thermo()
    for k in ("temp", "pair_pe", "pressure"):
        np.testing.assert_allclose(th[k], o["thermo"][k], rtol=1e-9, atol=1e-9)
    e.close()
