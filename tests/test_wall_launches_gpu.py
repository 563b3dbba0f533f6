"""fix two_wall and compute wall_contact with the small-grid launches (the step's bookkeeping in
the reflection's last block) and without: the wall extents are taken once a step and reset for
the next one in both, over runs cut at any step and beside a replica without walls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [(12,), (5, 1, 6)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_wall_channel_launches_agree(mode, runs):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.wall_channel(L=6.0, Lz=10.0, seed=81, dt=0.02, thermo=1, nsteps=12)
    out = []
    for m in (1, mode):
        e = Engine(s.run_in, system=s.c_system())
        e.set_tuning(launch_mode=m)
        for n in (12,) if m == 1 else runs:
            e.run(n)
        out.append((e.thermo(), e.state(), e.compute("cwc")))
        e.close()
    (ta, sa, ca), (tb, sb, cb) = out
    assert list(tb["step"]) == list(range(13))
    # FP32 force sums in another order: 1e-7 of the force, grown over 0.24 time units
    np.testing.assert_allclose(tb["temp"], ta["temp"], rtol=1e-5)
    liquid = s.types == 1
    walls_lo, walls_hi = sa["x"][s.types == 2, 2].max(), sa["x"][s.types == 3, 2].min()
    for st in (sa, sb):
        assert st["x"][liquid, 2].min() >= walls_lo - 1e-5 and st["x"][liquid, 2].max() <= walls_hi + 1e-5
    assert np.abs(sa["v"] - sb["v"]).max() < 5e-4
    np.testing.assert_array_equal(ca[:, 0], cb[:, 0])
    assert np.abs(ca[:, 1] - cb[:, 1]).max() <= 1


def test_wall_channel_in_a_batch():
    from gpumdpd_b200 import Batch, Engine, inputs
    s = inputs.wall_channel(L=6.0, Lz=10.0, seed=82, dt=0.02, thermo=1, nsteps=6)
    q = inputs.plain_dpd(L=5.0, seed=83, dt=0.02, thermo=1, nsteps=6)
    b = Batch([q.run_in, s.run_in], [q.c_system(), s.c_system()])
    b.run(6)
    e = Engine(s.run_in, system=s.c_system())
    e.run(6)
    np.testing.assert_allclose(b.thermo(1)["temp"], e.thermo()["temp"], rtol=1e-5)
    b.close()
    e.close()
