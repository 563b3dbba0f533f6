"""The launches and the pair kernel that bench.py reports (no GPU), against the launch lists of the
default step: 11 kernels on the 3M melt, 6 on 3000 particles (profiles/launches_*.md)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


class _Sys:
    def __init__(self, n, box, run_in="neighbor 1.0 0.0 10.0 1\npair_style dpd 1.0 1.0 3\n"):
        self.n, self.box, self.run_in = n, np.full(3, float(box)), run_in


@pytest.mark.parametrize("n,box,want,kernel", [
    (3000, 10.0, 6, "k_pair_entry"),         # one scan block, tiny grid
    (24000, 20.0, 7, "k_pair_flat "),        # two scan launches; too many list entries for a thread each
    (192000, 40.0, 7, "k_pair_flat "),
    (648000, 60.0, 11, "k_pair_flat_split"),
    (3000000, 100.0, 11, "k_pair_flat_split"),
    (3000, 165.0, 8, "k_pair_entry"),        # more than 1024 scan blocks: three scan launches
])
def test_launches_of_a_step(n, box, want, kernel):
    import bench
    s = _Sys(n, box)
    assert bench.build_launches(s, 0.0) + bench.step_launches(s, 8) == want
    assert bench.pair_kernel_name(s, 8).startswith(kernel)


def test_launches_of_the_many_body_slab():
    import bench
    s = _Sys(33600, 30.0, "neighbor 1.0 0.3 20.0 1\npair_style mdpd 1.0 1.0 3\n")
    assert bench.step_launches(s, 8) == bench.step_launches(s, 11) == 3
    assert bench.list_capacity(s) == 192  # 20 * 4/3 pi 1.3^3 = 184
