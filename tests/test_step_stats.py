"""The statistics of a split step (maxima of |a|^2, ion fraction and the rates of A_nl) do not depend on the
step's length, down to a step of none."""
import numpy as np
import pytest

from mpc_gb300 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plasm", [0, 1])
def test_statistics_of_short_steps(gpu_lib, plasm):
    from mpc_gb300.capi import Propagator
    p, A = inputs.make_cell(inputs.cell64(Nx=32, Ny=32, Nt=256, energy=2e-3, plasm=plasm))
    got = {}
    with Propagator(p) as prop:
        st = prop.state()
        for dz in (1e-6, 1e-20, 1e-30, 0.0):
            prop.upload(A, calibrate=True)
            before = prop.download()
            st.dzz, st.z, st.nstep = dz, 0.0, 0
            prop.set_state(st)
            prop.step_stats(reset=True)
            prop.run_fixed(1)
            got[dz] = prop.step_stats(reset=True)
            if dz < 1e-6:   # nothing but the transforms' rounding
                assert np.linalg.norm(prop.download() - before) / np.linalg.norm(before) < 1e-6
    ref = got[1e-6]
    assert ref[0] > 0 and ref[2] > 0 and ref[3] > 0 and (ref[1] > 0) == bool(plasm)
    for dz, s in got.items():   # FP32 rates of fields that differ by the rounding of a step
        assert np.allclose(s, ref, rtol=1e-4), (dz, s, ref)
