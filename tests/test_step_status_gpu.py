"""A status raised by the integrate on a step without thermo outlives the step's bookkeeping, which
another block of the same launch does on small grids.

The list is checked every 50 steps only, so no list build after the first sees the non-finite
state, and no thermo row is due in the run: what the integrate raises is the only report.
Grids of one block, of several, and of a launch per part (above 148 x 8 blocks of 256 slots).
"""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DPD_E_NUMERIC = -7


@pytest.mark.parametrize("L", [4.0, 8.0, 20.0, 47.0])
@pytest.mark.parametrize("which", [0, 0.5, 1])
def test_nonfinite_velocity_without_thermo(L, which):
    from gpumdpd_b200 import Engine, capi, inputs
    s = inputs.plain_dpd(L=L, seed=7, skin=0.3, dt=0.01, nsteps=10, thermo=100000)
    run_in = s.run_in
    run_in = re.sub(r"(?m)^(neighbor \S+ \S+ \S+) \S+$", r"\1 50", run_in)
    e = Engine(run_in, system=s.c_system())
    e.run(3)
    st = e.state()
    v = st["v"].copy()
    v[int(which * (s.n - 1)), 1] = np.nan
    e.set_state(st["x"], v)
    with pytest.raises(capi.DpdError) as ex:
        e.run(2)
    assert ex.value.code == DPD_E_NUMERIC, str(ex.value)
    e.close()
