"""The counting sort over more than 1024 blocks of 4096 cells, where the block sums are scanned by a
launch of their own: a sparse box of 165 x 165 x 165 cells against the oracle's pair set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])  # the parity flip in the permutation or in a launch of its own
def test_scan_of_more_than_1024_blocks(oracle_mod, mode):
    from gpumdpd_b200 import Engine, inputs
    s = inputs.plain_dpd(L=165.3, rho=0.012, seed=62, dt=0.02, nsteps=5, skin=0.0)
    e = Engine(s.run_in, system=s.c_system())
    e.set_tuning(launch_mode=mode)
    e.run(2)
    c = e.cells()
    assert np.prod(c["nc"].astype(np.int64)) > 1024 * 4096
    got = e.neighbors()
    ref = oracle_mod.pairs_f32(np.arange(1, s.n + 1), c["cell"], c["offset"], c["nc"], c["w"], c["cut2"])
    assert len(got) == len(set(map(tuple, got.tolist()))) > 100
    assert set(map(tuple, got.tolist())) == set(map(tuple, ref.tolist()))
    e.close()
