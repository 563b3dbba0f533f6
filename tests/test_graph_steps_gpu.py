"""Runs that are cut into launches of several steps and of one: the same trajectory whatever the
run lengths, up to FP32 summation order, and the same step counters, rows and list builds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(17,), (1,) * 17, (7, 9, 1), (8, 8, 1), (0, 16, 1)])
def test_run_lengths_give_the_same_steps(lengths):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.diblock_melt(L=8.0, seed=71, dt=0.01, nsteps=17, thermo=1, skin=0.0)
    e = Engine(s.run_in, system=s.c_system())
    for n in lengths:
        e.run(n)
    ref = Engine(s.run_in, system=s.c_system())
    ref.run(17)
    a, b = e.thermo(), ref.thermo()
    assert list(a["step"]) == list(range(18)) == list(b["step"])
    assert e.info()["step"] == ref.info()["step"] == 17
    assert e.info()["builds"] == ref.info()["builds"] == 18  # skin 0: one per evaluation
    sa, sb = e.state(), ref.state()
    # FP32 force sums in another order (1e-7 of the RMS force) grow by less than e^5 per time
    # unit of this system, over 0.17 units; the largest of 4608 components
    assert np.abs(sa["v"] - sb["v"]).max() < 2e-5
    np.testing.assert_allclose(a["temp"], b["temp"], rtol=1e-5)
