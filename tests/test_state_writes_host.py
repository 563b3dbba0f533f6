"""No kernel stores a whole RepState (no GPU): its status word collects bits that any thread of a
launch may raise, so a store of the struct, which carries the word as it was read, can lose them.
When that happens depends on which thread comes first, and a run that shows it is rare."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpumdpd_b200", "csrc")


def test_no_kernel_stores_a_whole_replica_state():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for k, line in enumerate(open(path), 1):
            if re.search(r"\brstate\[[^\]]*\]\s*=[^=]|\bst\[[^\]]*\]\.status\s*=[^=]|rstate\[[^\]]*\]\.status\s*=[^=]", line):
                found.append(f"{os.path.basename(path)}:{k}: {line.strip()}")
    assert not found, found
