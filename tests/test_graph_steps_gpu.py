"""Runs that are cut into launches of several steps and of one: the same trajectory whatever the
run lengths, up to FP32 summation order, and the same step counters, rows and list builds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(24,), (1,) * 24, (7, 9, 8), (8, 8, 8), (0, 16, 8)])
def test_run_lengths_give_the_same_steps(lengths):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.diblock_melt(L=8.0, seed=71, dt=0.001, nsteps=136, thermo=1, skin=0.0, max_rho=15.0)
    e, ref = (Engine(s.run_in, system=s.c_system()) for _ in range(2))
    for eng, rest in ((e, lengths), (ref, (1,) * 24)):
        eng.run(112)  # launches of several steps begin after this
        for n in rest:
            eng.run(n)
    a, b = e.thermo(), ref.thermo()
    assert list(a["step"]) == list(range(137)) == list(b["step"])
    assert e.info()["step"] == ref.info()["step"] == 136
    assert e.info()["builds"] == ref.info()["builds"] == 137  # skin 0: one per evaluation
    sa, sb = e.state(), ref.state()
    # FP32 force sums in another order (1e-7 of the RMS force) grow by less than e^5 per time
    # unit of this system, over 0.14 units; the largest of 4608 components
    assert np.abs(sa["v"] - sb["v"]).max() < 2e-5
    np.testing.assert_allclose(a["temp"], b["temp"], rtol=1e-5)
