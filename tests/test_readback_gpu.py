"""State and thermo read-back: rows gathered by tag on the device against the slots read
through the cell representation, and thermo rows around the staged row count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [4.0, 6.0, 9.5])  # 192, 648, 2572 particles: below, across and at ragged ends of a block
def test_state_rows_by_tag(L):
    from gpumdpd_b200 import Engine, capi, inputs
    s = inputs.plain_dpd(L=L, seed=77, nsteps=10)
    e = Engine(s.run_in, system=s.c_system())
    v = s.v.astype(np.float32).astype(np.float64)
    e.set_state(s.x, v)
    e.run(0)  # forces of step 0 and the first cell sort: velocities stay
    st = e.state()
    np.testing.assert_array_equal(st["v"], v)
    # half a float ulp of a cell offset (< 2), and the box of float cell widths
    assert np.abs(st["x"] - s.x).max() < 1.2e-7 + 1.2e-7 * L
    e.run(7)
    st, c = e.state(), e.cells()
    box = c["nc"].astype(np.float64) * c["w"].astype(np.float64)
    x = c["cell"].astype(np.float64) * c["w"].astype(np.float64) + c["offset"].astype(np.float64)
    x = x - np.floor(x / box) * box
    np.testing.assert_array_equal(st["x"], x)
    # any subset of the arrays gives the same rows
    lib = capi.load()
    for want in ((0, 1, 0, 1), (1, 0, 0, 0), (0, 0, 1, 0)):
        out = [np.full((s.n, 3), -7.0), np.full((s.n, 3), -7.0), np.full((s.n, 3), -7, dtype=np.int32),
               np.full((s.n, 3), -7.0)]
        assert lib.dpd_get_state(e.h, *(capi.ptr(a) if w else None for a, w in zip(out, want))) == 0
        for a, w, k in zip(out, want, ("x", "v", "image", "f")):
            np.testing.assert_array_equal(a, st[k] if w else np.full_like(a, -7))
    e.close()


def test_thermo_rows_staged_or_not():
    from gpumdpd_b200 import Engine, inputs
    s = inputs.plain_dpd(L=4.0, seed=78, nsteps=10, thermo=1)
    e = Engine(s.run_in, system=s.c_system())
    e.run(3)
    assert list(e.thermo(64)["step"]) == [0, 1, 2, 3]
    assert list(e.thermo(65)["step"]) == [0, 1, 2, 3]
    e.run(2060)  # past the 2048 rows that the device keeps
    every = e.thermo(4096)
    assert list(every["step"]) == list(range(16, 2064))
    for n in (1, 63, 64, 65, 200):
        t = e.thermo(n)
        for k in every:
            np.testing.assert_array_equal(t[k], every[k][-n:])
    e.close()
