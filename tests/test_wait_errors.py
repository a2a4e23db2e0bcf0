"""A wait that ran out in a kernel is reported by whichever call next returns something of the field or
decides on it.  The wait is the library's own probe (bounded, about a second), queued on the context's
stream before the call."""
import ctypes as C

import numpy as np
import pytest

from mpc_gb300 import inputs

pytestmark = pytest.mark.gpu


def _linearstep(prop, A, batch):
    one = np.ones(prop.p.Nt, dtype=np.complex128)
    prop.linearstep(A, one, np.ones(prop.p.Nx, dtype=np.complex128))


CALLS = {
    "ssfmprop": lambda prop, A, batch: prop.ssfmprop(A, prop.p.dzz, 1, 0.0, prop.p.puls_e),
    "ssfmprop with diagnostics": lambda prop, A, batch: prop.ssfmprop(A, prop.p.dzz, 1, 0.0, prop.p.puls_e, change=1),
    "linearstep": _linearstep,
    "step_double": lambda prop, A, batch: prop.step_double(),
    "batch run_fixed": lambda prop, A, batch: batch.run_fixed(2),
    "batch step_double": lambda prop, A, batch: batch.step_double(),
    "diag": lambda prop, A, batch: prop.diag(),
    "energy": lambda prop, A, batch: prop.energy(),
    "step_stats": lambda prop, A, batch: prop.step_stats(),
    "features": lambda prop, A, batch: prop.features(),
    "download": lambda prop, A, batch: prop.download(),
    "sync": lambda prop, A, batch: prop.sync(),
}


@pytest.mark.parametrize("name", CALLS)
def test_next_call_reports_a_wait_that_ran_out(gpu_lib, name):
    from mpc_gb300.capi import Batch, MPCError, Propagator
    p, A = inputs.make_cell(inputs.cell64(Nx=16, Ny=16, Nt=64))
    with Propagator(p) as prop, Propagator(p) as other:
        prop.upload(A, calibrate=True)
        other.upload(A, calibrate=True)
        batch = Batch([other, prop])
        prop.run_fixed(1)
        prop.sync()
        z, attempts = prop.state().z, prop.state().attempts
        assert gpu_lib.mpc_wait_limit_start(prop.h) == 0
        with pytest.raises(MPCError, match="MPC_ERR_TIMEOUT"):
            CALLS[name](prop, A.copy(), batch)
        if "step_double" in name:   # neither accepted nor rejected
            assert prop.state().z == z and prop.state().attempts == attempts
        prop.sync()                 # reported once, then cleared
        other.sync()
        CALLS[name](prop, A.copy(), batch)
        batch.close()


def test_null_context_is_refused(gpu_lib):
    assert gpu_lib.mpc_wait_limit_start(None) == 1   # MPC_ERR_ARG
