"""The FP64 engine in boxes of mostly empty cells, where it takes the forces with a warp per atom:
positions, velocities, forces, images and thermo rows against the FP64 oracle, and repeats bit for bit.

All boxes have enough cells for that pass (csrc/launch_rules.h, atom_pass); tolerances are those of the
engine's other oracle tests: only FP64 summation order separates the two.
"""
import numpy as np
import pytest

from conftest import force_err

pytestmark = pytest.mark.gpu


def _system(name, thermo):
    from gpumdpd_b200 import inputs
    k = dict(seed=94, dt=0.02, nsteps=10, thermo=thermo, skin=0.0, max_rho=30.0)
    if name == "gas":
        return inputs.plain_dpd(L=45.3, rho=0.05, **k)
    if name == "half_full":  # a record or two in most occupied cells
        return inputs.plain_dpd(L=34.0, rho=0.5, **k)
    if name == "chains":
        return inputs.diblock_melt(L=45.3, rho=0.05, **k)
    if name == "angles":
        return inputs.angle_chains(L=45.3, rho=0.05, **k)
    if name == "half_integrated":
        s = inputs.binary_mixture(L=45.3, a_ab=40.0, rho=0.05, **k)
        s.run_in = s.run_in.replace("group all type 1 2", "group a type 1").replace("fix md all nve", "fix md a nve")
        assert "fix md a nve" in s.run_in
        return s
    if name == "many_body_drop":  # dense cells, several queues of pairs an atom, among empty ones
        return inputs.mdpd_slab(Lx=45.3, Ly=45.3, Lz=60.0, z0=20.0, z1=20.4, rho=6.0, rho_vapour=0.01,
                                **dict(k, dt=0.002))
    s = inputs.plain_dpd(L=60.0, rho=0.006, **dict(k, dt=0.002))  # "cube": 1296 atoms within 6 x 6 x 6
    rng = np.random.default_rng(3)
    x = rng.uniform(-3.0, 3.0, (s.n, 3)) % 60.0  # about the corner: every side of the box
    return inputs.System(s.lo, s.hi, s.masses, s.types, x, s.v, run_in=s.run_in)


@pytest.mark.parametrize("thermo", [100, 3])
@pytest.mark.parametrize("name", ["gas", "half_full", "chains", "angles", "half_integrated", "many_body_drop", "cube"])
def test_sparse_boxes_match_oracle(oracle_mod, name, thermo):
    from gpumdpd_b200 import Engine
    s = _system(name, thermo)
    e, again = (Engine(s.run_in, system=s.c_system(), precision="fp64") for _ in range(2))
    ff = oracle_mod.ff_from_run_in(s.run_in, s.masses)
    box = s.hi - s.lo
    done = 0
    for n in (3, 1, 4):
        e.run(n)
        again.run(n)
        done += n
        st = e.state()
        oracle_mod.set_saru_double_tail(True)
        try:
            o = oracle_mod.run(ff, np.arange(1, s.n + 1), s.types, s.x, s.v, s.lo, box, 1, done, thermo,
                               bonds=s.bonds, angles=getattr(s, "angles", None))
        finally:
            oracle_mod.set_saru_double_tail(False)
        dx = (st["x"] + st["image"] * box) - (o["x"] + o["image"] * box)
        assert np.abs(dx).max() < 1e-9
        assert np.abs(st["v"] - o["v"]).max() < 1e-9
        assert force_err(st["f"], o["f"]) < 1e-9
    assert np.abs(o["image"]).sum() > 0
    th = e.thermo()
    assert list(th["step"]) == [k for k in range(done + 1) if k % thermo == 0]
    for k in ("temp", "pair_pe", "bond_pe", "angle_pe", "pressure"):
        np.testing.assert_allclose(th[k], o["thermo"][k], rtol=1e-9, atol=1e-9)
    other = again.state()
    for k in ("x", "v", "f", "image"):
        np.testing.assert_array_equal(st[k], other[k])
    e.close()
    again.close()
