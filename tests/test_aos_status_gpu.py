"""A bad id or type anywhere in the AoS input is reported: the thread that sets the call's step
must not write over the status that other threads of the same launch raise.

Positions: the first entry (the thread that sets the step), the same warp, the first block, other
blocks, the last entry; each on fresh engines, several times, as which thread comes first is open.
The engine's state has left the L2 when the call begins and the ids and types are in it, so that the
thread that reads the state waits the longest.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DPD_E_ARG = -1
TRIES = 12


@pytest.mark.parametrize("what", ["id", "type"])
@pytest.mark.parametrize("where", [0, 1, 33, 257, 0.5, 1.0])
def test_one_bad_entry_is_reported(what, where):
    import torch
    from gpumdpd_b200 import DpdError, Engine, inputs
    s = inputs.plain_dpd(L=14.0, seed=12, nsteps=10)
    k = where if isinstance(where, int) else int(where * (s.n - 1))
    dev = torch.device("cuda")
    xd = torch.tensor(s.x.astype(np.float32).reshape(-1), device=dev)
    vd = torch.zeros(3 * s.n, device=dev)
    fd = torch.zeros(3 * s.n, device=dev)
    ids = torch.arange(1, s.n + 1, dtype=torch.int32, device=dev)
    types = torch.tensor(s.types, dtype=torch.int32, device=dev)
    (ids if what == "id" else types)[k] = s.n + 7
    flush = torch.zeros(1 << 28, dtype=torch.uint8, device=dev)  # twice the L2
    reported = 0
    for step in range(TRIES):
        e = Engine(s.run_in, system=s.c_system())
        flush += 1
        (ids + types).sum().item()
        try:
            e.pair_compute_aos(xd.data_ptr(), vd.data_ptr(), ids.data_ptr(), types.data_ptr(), s.n, step,
                               fd.data_ptr())
        except DpdError as ex:
            assert ex.code == DPD_E_ARG, str(ex)
            reported += 1
        e.close()
    assert reported == TRIES
