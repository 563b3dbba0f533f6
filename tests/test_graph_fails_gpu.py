"""A graph that cannot be made costs no state.  A child process runs an engine with
cudaGraphInstantiate replaced by a function that answers cudaErrorMemoryAllocation on chosen calls
(nothing on the GPU fails).  A run that would use the graph of several steps goes on with the one of a
single step; time_steps, which needs its own graph, returns the error before the first drift.  Either
way the steps that follow are those of an engine that never met the error."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>
int cudaGraphInstantiate(void** exec, void* graph, unsigned long long flags)
{
    static int call;
    static int (*real)(void**, void*, unsigned long long);
    const char* fail = getenv("FAIL_CALL");
    if (++call == (fail ? atoi(fail) : 0)) return 2;
    if (!real) real = dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaGraphInstantiate");
    return real(exec, graph, flags);
}
"""

CHILD = r"""
import sys
import numpy as np
from gpumdpd_b200 import DpdError, Engine, inputs
what, fail, out = sys.argv[1:]
s = inputs.diblock_melt(L=8.0, seed=71, dt=0.001, nsteps=200, thermo=1, skin=0.0, max_rho=15.0)
e = Engine(s.run_in, system=s.c_system())
e.run(112)
raised = 0
if what == "time" and fail != "0":
    try:
        e.time_steps(4)
    except DpdError as ex:
        assert ex.code == -4, ex.code
        raised = 1
try:
    e.run(20)
except DpdError as ex:
    raised = 2
    e.run(20)
e.run(12)
st, th, info = e.state(), e.thermo(), e.info()
np.savez(out, x=st["x"], v=st["v"], rows=th["step"], step=info["step"], builds=info["builds"], raised=raised)
e.close()
"""


def _child(tmp_path, shim, what, fail):
    out = str(tmp_path / f"{what}{fail}.npz")
    env = dict(os.environ, LD_PRELOAD=shim, FAIL_CALL=str(fail), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, what, str(fail), out], env=env, cwd=ROOT, timeout=120,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(out)


@pytest.mark.parametrize("what", ["run", "time"])
def test_failed_graph_leaves_the_steps_as_they_are(tmp_path, what):
    (tmp_path / "shim.c").write_text(SHIM)
    shim = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", shim, str(tmp_path / "shim.c"), "-ldl"], check=True)
    ref = _child(tmp_path, shim, what, 0)
    got = _child(tmp_path, shim, what, 2)  # call 1: the graph that an engine is created with
    assert ref["raised"] == 0 and got["raised"] == (1 if what == "time" else 0)
    assert got["step"] == ref["step"] == 144
    assert got["builds"] == ref["builds"] == 145  # skin 0: one per evaluation
    assert list(got["rows"]) == list(ref["rows"]) == list(range(145))
    # FP32 force sums in another order (1e-7 of the RMS force), grown over 0.15 time units, as for
    # runs cut into launches of different lengths
    assert np.abs(got["v"] - ref["v"]).max() < 2e-5
