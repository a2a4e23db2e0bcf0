"""The split-step pencil kernel (mpc_step.cuh) against the FP64 oracle where its branches part: every
transform length (its radix plans and warp layouts differ), both field layouts, and fields strong enough
for the second ionization stage, for exponents beyond the series of exp and sin/cos, and for an ion
fraction beyond the series of 1 - exp(-R).

Tolerance: one split step in FP32 reproduces the FP64 step to about 1e-6 relative (the 1e-5 of the
other single-step checks); a nonlinear phase of a few rad multiplies its own rounding, 1e-7, by that."""
import numpy as np
import pytest

import oracle
from mpc_gb300 import inputs

pytestmark = pytest.mark.gpu

# energy [J], gas, pressure [bar], step [m]
WEAK = (0.5e-3, "Argon", 1.0, 2e-3)
SECOND = (30e-3, "Argon", 0.2, 2e-3)      # |a|^2 about 170: second-stage probabilities above 2^-60
PHASE = (3e-3, "Argon", 3.0, 3e-2)        # Kerr phase about 0.9 rad per step
IONIZED = (60e-3, "Krypton", 0.02, 1e-3)  # first stage saturated: R well above 1/8

GRIDS = [(16, 64, 0), (32, 256, 0), (64, 512, 0), (128, 1024, 0), (256, 2048, 3), (256, 2048, 9)]


def _one_step(n, nt, variant, energy, gas, bar, dz, **kw):
    from mpc_gb300.capi import Propagator
    p, A = inputs.make_cell(inputs.cell64(Nx=n, Ny=n, Nt=nt, window_xy=3e-3, window_t=1e-12, beam_w=0.3e-3, fwhm=120e-15,
                                          energy=energy, gas=gas, pressure=bar, **kw))
    o = oracle.Oracle(p)
    o.calibrate(A)
    ref = A.copy()
    o.ssfmprop(ref, dz, 1, 0.0, p.puls_e)
    with Propagator(p.copy(variant=variant)) as prop:
        got = A.copy()
        prop.ssfmprop(got, dz, 1, 0.0, p.puls_e)
    return float(np.linalg.norm(got - ref) / np.linalg.norm(ref)), float(np.abs(ref).max() / np.abs(A).max())


@pytest.mark.parametrize("n,nt,variant", GRIDS)
@pytest.mark.parametrize("case", [WEAK, SECOND, PHASE, IONIZED])
def test_one_step_matches_oracle(gpu_lib, n, nt, variant, case):
    if nt >= 1024 and case in (WEAK, PHASE):
        pytest.skip("covered by the production-grid checks")
    err, _ = _one_step(n, nt, variant, *case)
    assert err < 1e-5


@pytest.mark.parametrize("n,nt", [(16, 64), (32, 256), (64, 512), (128, 1024)])
@pytest.mark.parametrize("plasm,sst", [(0, 1), (1, 0), (0, 0)])
def test_switched_off_terms(gpu_lib, n, nt, plasm, sst):
    err, _ = _one_step(n, nt, 0, *PHASE, plasm=plasm, sst_on=sst)
    assert err < 1e-5


@pytest.mark.parametrize("n,nt", [(16, 64), (16, 256), (64, 512), (64, 1024), (16, 2048)])
@pytest.mark.parametrize("plasm,sst", [(1, 1), (0, 1), (1, 0), (0, 0)])
def test_nonlinear_noalloc_alignment_and_terms(gpu_lib, n, nt, plasm, sst):
    """The allocation-free nonlinear step with each term switched off, on a 16-byte aligned field and on
    one that is only 8-byte aligned (element-wise tile loads: the same values), against the oracle;
    64x64x512 and 64x64x1024 give some CTAs more than one tile."""
    torch = pytest.importorskip("torch")
    from mpc_gb300.capi import nonlinear_noalloc
    p, A = inputs.make_cell(inputs.cell64(Nx=n, Ny=n, Nt=nt, window_xy=3e-3, window_t=1e-12, beam_w=0.3e-3, fwhm=120e-15, energy=3e-3,
                                          pressure=3.0, plasm=plasm, sst_on=sst))
    p = p.copy(betas=np.zeros(nt), wr=np.zeros(n), alpha=0.0)
    o = oracle.Oracle(p)
    o.calibrate(A)
    dz = 3e-2
    out = []
    for off in (0, 1):
        buf = torch.zeros(A.size + 2, dtype=torch.complex64, device="cuda")
        dev = buf[off:off + A.size]
        dev.copy_(torch.from_numpy(A.astype(np.complex64)))
        assert dev.data_ptr() % 16 == 8 * off
        assert nonlinear_noalloc(p, dev.data_ptr(), dz, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        out.append(dev.cpu().numpy())
        assert buf[A.size + off:].abs().max() == 0 and buf[:off].abs().sum() == 0
    assert np.array_equal(out[0], out[1])
    ref = A.copy()
    o.ssfmprop(ref, dz, 1, 0.0, p.puls_e)
    assert np.linalg.norm(out[0] - ref) / np.linalg.norm(ref) < 1e-5


@pytest.mark.parametrize("n,nt,variant", [(16, 64, 0), (32, 256, 0), (64, 512, 0), (128, 1024, 0), (256, 512, 0), (256, 2048, 3)])
def test_diagnostics_match_numpy(gpu_lib, n, nt, variant):
    """The one-sweep diagnostics (temporal profile, spectrum, beam profiles) of a random field, several
    tiles per CTA at the larger grids, against numpy in FP64 (FP32 transforms and runs of 32: 1e-6)."""
    from mpc_gb300.capi import Propagator
    p, A = inputs.make_cell(inputs.cell64(Nx=n, Ny=n, Nt=nt, noise=0.0))
    rng = np.random.default_rng(nt)
    A = np.abs(A).max() * (A.reshape(nt, n, n) + 0.3 * (rng.standard_normal((nt, n, n)) + 1j * rng.standard_normal((nt, n, n))))
    with Propagator(p.copy(variant=variant)) as prop:
        prop.upload(A.reshape(-1))
        got = prop.diag()
        again = prop.diag()
    I = np.abs(A) ** 2
    ref = (I.sum(axis=(1, 2)), (np.abs(np.fft.fft(A, axis=0)) ** 2).sum(axis=(1, 2)), I.sum(axis=(0, 1)), I.sum(axis=(0, 2)))
    for g, h, r in zip(got, again, ref):
        assert np.linalg.norm(g - r) / np.linalg.norm(r) < 1e-6
        assert np.allclose(g, h, rtol=1e-12)


def test_boundary_conversions(gpu_lib):
    """Download converts to complex128 without FP64 instructions: a field of one sample per pencil shows the
    conversions.  Values over the whole range of
    physical fields, zeros, powers of two, tiny, huge and negative ones: within FP32 rounding of the
    transforms; zeros exactly."""
    from mpc_gb300.capi import Propagator
    p, _ = inputs.make_cell(inputs.cell64(Nx=32, Ny=32, Nt=256))
    rng = np.random.default_rng(2)
    A = np.zeros((256, 1024), dtype=np.complex128)
    mag = 10.0 ** rng.uniform(-30, 20, 1024)
    mag[::9] = np.ldexp(1.0, rng.integers(-60, 60, mag[::9].size))
    mag[::31] = 0.0
    A[5] = mag * np.exp(2j * np.pi * rng.integers(0, 8, 1024) / 8)
    with Propagator(p) as prop:
        prop.upload(A.reshape(-1))
        got = prop.download().reshape(256, 1024)
    ref = np.abs(A).max(axis=0)
    err = np.abs(got - A).max(axis=0)
    assert np.all(err[ref == 0] == 0)
    # 8 stages forward and back of 256 points, each within 2^-23 of its values (a sample spread over 256)
    big = ref > 1e-15          # smaller ones leave FP32's normal range in device units
    assert np.all(err[big] < 2e-6 * ref[big]) and np.all(np.isfinite(got))
    A[5, :] = 0
    A[:, 0] = np.nan
    with Propagator(p) as prop:
        prop.upload(A.reshape(-1))
        got = prop.download().reshape(256, 1024)
    assert np.isnan(got[:, 0]).all() and not got[:, 1:].any()
