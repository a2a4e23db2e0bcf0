"""Identical calls give identical bits where no sum depends on the order in which CTAs finish: the
diagnostics' four profiles, and the beam profiles of a step-doubling attempt."""
import numpy as np
import pytest

from mpc_gb300 import inputs

pytestmark = pytest.mark.gpu

# several tiles per CTA and CTAs per SM; one part of the rows (Nt = 64) and several; both field layouts
GRIDS = [(16, 64, 0), (64, 512, 2), (128, 1024, 5), (256, 512, 0), (256, 512, 5), (256, 2048, 3)]


def _field(n, nt):
    p, A = inputs.make_cell(inputs.cell64(Nx=n, Ny=n, Nt=nt, noise=0.0))
    rng = np.random.default_rng(n + nt)
    return p, (A * (1.0 + 0.3 * rng.standard_normal(A.size))).astype(np.complex128)


@pytest.mark.parametrize("n,nt,variant", GRIDS)
def test_diagnostics_repeat(gpu_lib, n, nt, variant):
    from mpc_gb300.capi import Propagator
    p, A = _field(n, nt)
    with Propagator(p.copy(variant=variant)) as prop:
        prop.upload(A, calibrate=True)
        first = prop.diag()
        for _ in range(8):
            assert all(np.array_equal(a, b) for a, b in zip(prop.diag(), first))


@pytest.mark.parametrize("n,nt,variant", GRIDS[:5])
def test_step_doubling_profiles_repeat(gpu_lib, n, nt, variant):
    from mpc_gb300.capi import Propagator
    p, A = _field(n, nt)
    with Propagator(p.copy(variant=variant)) as prop:
        st = prop.state()
        got = []
        for _ in range(6):
            prop.upload(A, calibrate=True)
            prop.set_state(st)
            r = prop.step_double(profiles=True)
            got.append(r)
        for r in got[1:]:
            assert np.array_equal(r["BP1"], got[0]["BP1"]) and np.array_equal(r["BP2"], got[0]["BP2"])
