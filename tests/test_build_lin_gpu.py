"""The list build under the linear cell order (slot ranges of whole columns, hits kept as bits)
where its ranges can go wrong, and the counting sort's scan over one and several blocks of
cells: the oracle's pair set, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(oracle_mod, e, n):
    c = e.cells()
    got = e.neighbors()
    ref = oracle_mod.pairs_f32(np.arange(1, n + 1), c["cell"], c["offset"], c["nc"], c["w"], c["cut2"])
    assert len(got) == len(set(map(tuple, got.tolist())))
    assert set(map(tuple, got.tolist())) == set(map(tuple, ref.tolist()))


# launch mode 1: a thread per slot; 0: one per slot and column group.
# boxes of 3 cells (a column is 3 cells, both ends wrap), ranges of more than 32 and of exactly
# few slots, empty cells, a last cell that ends with the slots
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("L,rho,skin", [(3.0, 3.0, 0.0), (3.1, 14.0, 0.0), (5.3, 9.0, 0.3), (8.2, 0.5, 0.0),
                                        (9.9, 3.0, 0.3), (6.0, 40.0, 0.0)])
def test_linear_build_gives_the_oracle_pairs(oracle_mod, L, rho, skin, mode):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.plain_dpd(L=L, rho=rho, seed=61, dt=0.005, nsteps=5, skin=skin, max_rho=80.0)
    e = Engine(s.run_in, system=s.c_system())
    e.set_tuning(launch_mode=mode)
    e.run(0)
    _check(oracle_mod, e, s.n)
    if skin == 0.0:  # a list every step, of that step's positions
        e.run(3)
        _check(oracle_mod, e, s.n)
    e.close()


@pytest.mark.parametrize("L", [15.9, 16.0, 17.3, 26.2])  # 3375, 4096, 4913 and 17576 cells and a ghost cell
def test_scan_over_blocks_of_cells(oracle_mod, L):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.plain_dpd(L=L, rho=0.7, seed=62, dt=0.005, nsteps=5, skin=0.0)
    e = Engine(s.run_in, system=s.c_system())
    e.set_tuning(launch_mode=1)
    e.run(2)
    _check(oracle_mod, e, s.n)
    e.close()


def test_aos_call_between_cell_orders(oracle_mod):
    """The AoS entry after a changed cell order that no run has uploaded yet still builds the
    right list (it keeps the old ranks)."""
    import torch
    from conftest import force_err
    from gpumdpd_b200 import Engine, inputs
    s = inputs.plain_dpd(L=8.0, seed=63, nsteps=5, skin=0.0)
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    x, v = s.x.astype(np.float32), s.v.astype(np.float32)
    for order, then in ((1, 0), (0, 1), (2, 0), (0, 0)):
        e = Engine(s.run_in, system=s.c_system())
        e.set_tuning(cell_order=order, launch_mode=1)
        e.run(0)
        e.set_tuning(cell_order=then, launch_mode=1)
        c = e.cells()
        L = c["nc"].astype(np.float64) * c["w"].astype(np.float64)
        dev = [torch.tensor(a.reshape(-1), device="cuda") for a in (x, v)]
        ids = torch.arange(1, s.n + 1, dtype=torch.int32, device="cuda")
        types = torch.tensor(s.types, dtype=torch.int32, device="cuda")
        f = torch.zeros(3 * s.n, device="cuda")
        e.pair_compute_aos(dev[0].data_ptr(), dev[1].data_ptr(), ids.data_ptr(), types.data_ptr(), s.n, 4, f.data_ptr())
        o = oracle_mod.forces(ff, np.arange(1, s.n + 1), s.types, x.astype(np.float64), v.astype(np.float64), s.lo, L, 4)
        assert force_err(f.cpu().numpy().reshape(-1, 3), o["f"]) < 1e-5
        e.close()
