"""What is timed: the propagator's work as a program that uses it has it done, one case per kind of call.

Every case goes through the public entry points of mpc_gb300.capi.  The field on the device is complex64,
and the boundary's complex128 values hold no more than that, so a case keeps its results in single
precision: fields as complex64, sums over a field (profiles, spectra) as float32 in SI units.  A field
that comes back to the host is taken on to the GPU as a torch tensor, where a program that post-processes
it has it.

`exact` states the same operators in torch, in 64 bits: the symmetric split step (dispersion, diffraction,
Kerr, self-steepening, ADK ionization, plasma), the step-doubling attempt, the diagnostics and the
controller network's training.
"""
import math

import numpy as np
import torch

# constants of the physical model (SI, and the atomic units of the ionization rates)
C0, HBAR, ME, EL0, EPS0 = 299792458.0, 1.054560652926899e-34, 9.1094e-31, 1.602e-19, 8.8541878128e-12
ZW0, FCTR, IH, EF, NAVO, T0 = 377.0, 0.89, 27.21, 5.14220642e11, 6.02214e23, 2.4188843265e-17
LAM0, ROC, CAV = 1030e-9, 0.3, 0.5
# gas: first and second ionization potential [eV], density [g/m^3], molar mass [g/mol], collision cross-section [m^2]
GASES = {
    "Argon": (15.75962, 27.62967, 1.784e3, 39.941, 1.57e-20),
    "Helium": (24.58741, 54.41778, 0.166e3, 4.002602, 6.11e-20),
    "Neon": (21.5646, 40.96328, 0.9002e3, 20.1797, 1.65e-20),
    "Krypton": (13.99961, 24.35985, 3.749e3, 83.798, 1.15e-20),
}
GRIDS = [(16, 64), (32, 256), (64, 512), (128, 1024), (256, 512), (256, 2048), (512, 1024)]  # (Nx = Ny, Nt)


def _cell(nx, ny, nt, **kw):
    c = {"nx": nx, "ny": ny, "nt": nt, "gas": "Argon", "bar": 1.0, "mj": 1.0, "fs": 250.0, "sst": 1, "plasma": 1, "lens": 1,
         "steps_per_pass": 400}
    c.update(kw)
    return c


def listed():
    return [
        # the reference's own call on its own kind of buffer (a host array), at the smallest grid: latency
        {"name": "dropin_16x16x64", "kind": "ssfm", "pinned": 0, "change": 1, **_cell(16, 16, 64, mj=0.05, steps_per_pass=50)},
        # the same call at an ordinary grid from page-locked buffers, with the beam profiles of an accepted step
        {"name": "dropin_128x128x1024", "kind": "ssfm", "pinned": 1, "change": 1, **_cell(128, 128, 1024, mj=0.5)},
        # one pass of the small cell (200 fixed steps, across a mirror): upload, run, download
        {"name": "fixed_64x64x512", "kind": "fixed", "steps": 200, "from": 100, **_cell(64, 64, 512, mj=0.2, steps_per_pass=200)},
        # a chunk of fixed steps of a sweep-sized cell, sign-flip mirror, another gas
        {"name": "fixed_128x128x1024", "kind": "fixed", "steps": 48, "from": 380, **_cell(128, 128, 1024, gas="Krypton", mj=0.6, lens=0)},
        # the other sweep grid without ionization (Kerr and self-steepening only)
        {"name": "fixed_256x256x512", "kind": "fixed", "steps": 40, "from": 0, **_cell(256, 256, 512, mj=0.4, plasma=0)},
        # half a pass of the large cell, across its mirror: the long device-resident run
        {"name": "fixed_256x256x2048", "kind": "fixed", "steps": 200, "from": 300, **_cell(256, 256, 2048)},
        # adaptive step doubling in the plasma-dominated cell
        {"name": "adaptive_512x512x1024", "kind": "adaptive", "attempts": 4, **_cell(512, 512, 1024, mj=3.0, fs=120.0, bar=3.0)},
        # a share of a parameter sweep: cells of both sweep grids advanced together
        {"name": "sweep_6_cells", "kind": "batch", "cells": 6, "steps": 16, **_cell(0, 0, 0)},
        # the diagnostics record of an accepted step: temporal profile, spectrum, beam profiles
        {"name": "diag_256x256x2048", "kind": "diag", **_cell(256, 256, 2048)},
        # the nonlinear step on a field that another program holds on the device, large
        {"name": "nonlinear_256x256x2048", "kind": "nonlinear", **_cell(256, 256, 2048)},
        # the same on a grid that is no power of two across
        {"name": "nonlinear_120x100x1024", "kind": "nonlinear", **_cell(120, 100, 1024, mj=2.0, fs=120.0, bar=2.0)},
        # one epoch of the step-size controller's training
        {"name": "train_16384", "kind": "train", "n": 16384, "batch": 256, "epochs": 1},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["ssfm", "fixed", "fixed", "adaptive", "batch", "diag", "nonlinear", "nonlinear", "train"])
    if kind == "train":
        return {"kind": "train", "n": int(_log(rng, 1000, 100000)), "batch": rng.choice([128, 256, 300, 512]), "epochs": 1}
    opts = {"gas": rng.choice(sorted(GASES)), "bar": round(rng.uniform(0.5, 3.0), 3), "mj": round(_log(rng, 0.1, 2.0), 4),
            "fs": round(rng.uniform(100, 300), 1), "sst": int(rng.random() < 0.8), "plasma": int(rng.random() < 0.8),
            "lens": rng.randrange(2), "steps_per_pass": rng.randrange(300, 500)}
    if kind == "batch":
        return {"kind": "batch", "cells": rng.randrange(2, 9), "steps": rng.randrange(4, 24), **_cell(0, 0, 0, steps_per_pass=opts["steps_per_pass"])}
    if kind == "nonlinear":
        nt = rng.choice([64, 256, 512, 1024, 2048])
        unit = 16384 // nt  # a tile of pencils: Nx Ny is a multiple of it
        nx = int(_log(rng, 12, 256))
        g = unit // math.gcd(nx, unit)
        ny = g * max(1, int(_log(rng, 12, 256)) // g)
        return {"kind": "nonlinear", **_cell(nx, ny, nt, **opts)}
    grids = [g for g in GRIDS if kind in ("fixed", "diag") or g[0] * g[0] * g[1] <= 1 << 25 or kind == "adaptive"]
    n, nt = rng.choice(grids)
    size = n * n * nt
    c = {"kind": kind, **_cell(n, n, nt, **opts)}
    if kind == "ssfm":
        c.update(pinned=rng.randrange(2), change=rng.randrange(2))
    if kind == "fixed":
        most = max(4, min(200, int(200 * 2**27 / size / 2)))
        c.update(steps=rng.randrange(3, most + 1), **{"from": rng.randrange(0, 300)})
    if kind == "adaptive":
        c.update(attempts=rng.randrange(1, 4 if size >= 1 << 27 else 9))
    return c


# ---- the physical set-up --------------------------------------------------------------------------
def _physics(c):
    """Grids and constants of a case's cell: x, y over 4 mm per 128 points at most 8 mm, t at 1 to 4 ps."""
    nx, ny, nt = c["nx"], c["ny"], c["nt"]
    n = max(nx, ny)
    window = 8e-3 if n >= 200 else 4e-3
    dx, dt = window / n, (1e-12 if nt <= 64 else 2e-12 if nt <= 1024 else 4e-12) / nt
    i1, i2, dens, mol, sig = GASES[c["gas"]]
    k0, w0 = 2 * math.pi / LAM0, 2 * math.pi * C0 / LAM0
    cent = lambda m: np.arange(m, dtype=np.float64) - m // 2  # noqa: E731
    w = 2 * np.pi * cent(nt) / (nt * dt)
    return {
        "nx": nx, "ny": ny, "nt": nt, "dx": dx, "dt": dt, "k0": k0, "w0": w0, "w": w, "x": cent(nx) * dx, "y": cent(ny) * dx,
        "t": cent(nt) * dt, "kx": 2 * np.pi * cent(nx) / (nx * dx), "ky": 2 * np.pi * cent(ny) / (ny * dx),
        "betas": 20e-27 * c["bar"] / 2 * w**2, "gamma2": 1e-23 * c["bar"] * k0 * HBAR * w0,
        "rho_nt": c["bar"] * dens * NAVO / mol, "rho_c": EPS0 * ME * w0**2 / EL0**2, "energy": c["mj"] * 1e-3, "beam": 0.5e-3,
        "fwhm": c["fs"] * 1e-15, "dz": CAV / c["steps_per_pass"], "gas": c["gas"], "sst": c["sst"], "plasma": c["plasma"],
        "lens": c["lens"], "i1": i1, "i2": i2, "sig": sig}


def _field(ph, seed):
    """(seed field on the GPU, complex128 [t, y, x], and its energy): a Gaussian pulse and beam, 1e-4 complex noise."""
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    t, y, x = (torch.from_numpy(ph[k]).to(dev) for k in "tyx")
    shape = (ph["nt"], ph["ny"], ph["nx"])
    a = torch.complex(torch.randn(shape, generator=g, device=dev), torch.randn(shape, generator=g, device=dev)).to(torch.complex128)
    a *= 1e-4 / math.sqrt(2.0)
    a += (torch.exp(-2 * math.log(2) * (t / ph["fwhm"]) ** 2)[:, None, None] * torch.exp(-((y / ph["beam"]) ** 2))[None, :, None]
          * torch.exp(-((x / ph["beam"]) ** 2))[None, None, :])
    esig = float(torch.view_as_real(a).square().sum()) * ph["dx"] ** 2 * ph["dt"] * HBAR * ph["w0"]
    return a, esig


def _params(ph, esig, variant, passes=8):
    from mpc_gb300.params import BOUNCE_LENS, BOUNCE_SIGNFLIP, MPCParams
    return MPCParams(dims=(ph["nx"], ph["ny"], ph["nt"]), dist=passes * CAV, dzz=ph["dz"], betas=ph["betas"], alpha=0.0, Cav=CAV, k0=ph["k0"],
                     wr=ph["ky"], sst_on=ph["sst"], w=ph["w"], gamma2=ph["gamma2"], w0=ph["w0"], plasm=ph["plasma"], deltat=ph["dt"],
                     rho_c=ph["rho_c"], rho_nt=ph["rho_nt"], n0=1.0, puls_e=ph["energy"], Ab_M=1.0, r=ph["y"], dr=ph["dx"], def_err=1e-5,
                     dzmin=1e-7, Esig=esig, gas=ph["gas"], bounce_mode=BOUNCE_LENS if ph["lens"] else BOUNCE_SIGNFLIP, roc=ROC,
                     variant=variant)


def _sweep(c, seed):
    """The cells of a share of a sweep: both grids in turn, pulse energy, gas pressure and duration spread."""
    r = np.random.default_rng(1000 + c["cells"])
    out = []
    for i in range(c["cells"]):
        n, nt = ((128, 1024), (256, 512))[i % 2]
        u = r.random(3)
        out.append((_cell(n, n, nt, mj=0.1 * 20 ** float(u[0]), bar=0.5 + 2.5 * float(u[1]), fs=100 + 200 * float(u[2]),
                          steps_per_pass=c["steps_per_pass"]), seed * 64 + i))
    return out


class _Resident:
    """A cell whose field lives on the device: its context and page-locked host buffers."""

    def __init__(self, c, seed, variant=-1, start=0):
        from mpc_gb300 import capi
        ph = _physics(c)
        a, esig = _field(ph, seed)
        n = a.numel()
        self.src = torch.empty(n, dtype=torch.complex128, pin_memory=True)
        self.src.copy_(a.reshape(-1))
        del a
        self.dst = torch.empty(n, dtype=torch.complex128, pin_memory=True)
        self.shape = (ph["nt"], ph["ny"], ph["nx"])
        self.prop = capi.Propagator(_params(ph, esig, variant))
        self.state0 = self.prop.state()
        self.state0.nstep = start
        self.state0.z = start * ph["dz"]

    def upload(self):
        self.prop.set_state(self.state0)
        self.prop.upload(self.src.numpy(), calibrate=True)

    def download(self):
        self.prop.download(self.dst.numpy())
        return self.dst.to("cuda", non_blocking=True).to(torch.complex64).reshape(self.shape)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "train":
        return _prepare_train(c, seed)
    if kind == "batch":
        from mpc_gb300 import capi
        cells = [_Resident(k, s) for k, s in _sweep(c, seed)]
        return {"c": c, "cells": cells, "batch": capi.Batch([x.prop for x in cells])}
    if kind in ("fixed", "adaptive"):
        return {"c": c, "cell": _Resident(c, seed, start=c.get("from", 0))}
    if kind == "diag":
        cell = _Resident(c, seed)
        cell.upload()
        cell.prop.sync()
        cell.src = cell.dst = None
        return {"c": c, "ph": _physics(c), "cell": cell}
    ph = _physics(c)
    a, esig = _field(ph, seed)
    a *= math.sqrt(ph["energy"] / esig)
    if kind == "nonlinear":
        a = a.to(torch.complex64)
        return {"c": c, "p": _params(ph, esig, 0), "dz": ph["dz"], "field": a, "work": torch.empty_like(a)}
    from mpc_gb300 import capi
    pin = bool(c["pinned"])
    field = torch.empty(a.numel(), dtype=torch.complex128, pin_memory=pin)
    field.copy_(a.reshape(-1))
    return {"c": c, "ph": ph, "field": field, "work": torch.empty(a.numel(), dtype=torch.complex128, pin_memory=pin),
            "prop": capi.Propagator(_params(ph, esig, 0))}


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "fixed":
        cell = s["cell"]
        cell.upload()
        cell.prop.run_fixed(c["steps"])
        return {"A": cell.download()}
    if kind == "adaptive":
        cell = s["cell"]
        cell.upload()
        bad = [cell.prop.step_double()["bad"] for _ in range(c["attempts"])]
        return {"A": cell.download(), "bad": np.array(bad), "dz": np.float32(cell.prop.state().dzz)}
    if kind == "batch":
        for cell in s["cells"]:
            cell.upload()
        s["batch"].run_fixed(c["steps"])
        return {"A": [cell.download() for cell in s["cells"]]}
    if kind == "diag":
        ph = s["ph"]
        temp, spec, bp1, bp2 = s["cell"].prop.diag()
        j = HBAR * ph["w0"]  # |A|^2 is a photon flux: power [W], spectral energy density [J s], fluence profiles [J/m]
        return {"temp": (temp * (j * ph["dx"] ** 2)).astype(np.float32), "spec": (spec * (j * (ph["dx"] * ph["dt"]) ** 2)).astype(np.float32),
                "BP1": (bp1 * (j * ph["dx"] * ph["dt"])).astype(np.float32), "BP2": (bp2 * (j * ph["dx"] * ph["dt"])).astype(np.float32)}
    if kind == "nonlinear":
        from mpc_gb300 import capi
        s["work"].copy_(s["field"])
        rc = capi.nonlinear_noalloc(s["p"], s["work"].data_ptr(), s["dz"], torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("nonlinear_noalloc: status %d" % rc)
        return {"A": s["work"]}
    if kind == "ssfm":
        ph, w = s["ph"], s["work"]
        w.copy_(s["field"])
        r = s["prop"].ssfmprop(w.numpy(), ph["dz"], 1, 0.0, ph["energy"], change=c["change"])
        out = {"A": w.to("cuda", non_blocking=True).to(torch.complex64)}
        if c["change"]:
            j = HBAR * ph["w0"] * ph["dx"] * ph["dt"]
            out.update(BP1=(r["BP1"] * j).astype(np.float32), BP2=(r["BP2"] * j).astype(np.float32))
        return out
    m = s["mlp"]
    m.weights = s["weights"]
    loss = m.train(s["X"], s["y"], epochs=c["epochs"], batch=c["batch"], lr=1e-3, seed=7)
    return {"weights": m.weights, "loss": np.float32(loss)}


# ---- work that a pass cannot do without -----------------------------------------------------------
def _step_work(c, host_bytes=0):
    """(bytes, flops) of one split step on a device field: two sweeps over a complex64 field, 5 n log2 n per transform,
    about 100 for the nonlinear step of a point with ionization, 40 without."""
    n = c["nx"] * c["ny"] * c["nt"]
    fft = 5 * (math.log2(c["nt"]) * (3 if c["sst"] else 2) + 2 * math.log2(c["nx"]) + 2 * math.log2(c["ny"]))
    return 32 * n, (fft + (100 if c["plasma"] else 40)) * n


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        per = 6 * (16 * 64 + 64 * 64 + 64)
        return {"bytes": 4 * 17 * c["n"] * c["epochs"], "flops": per * c["n"] * c["epochs"]}
    if kind == "batch":
        parts = [_step_work(k) for k, _ in _sweep(c, 0)]
        pts = sum(k["nx"] * k["ny"] * k["nt"] for k, _ in _sweep(c, 0))
        return {"bytes": 32 * pts + c["steps"] * sum(b for b, _ in parts), "flops": c["steps"] * sum(f for _, f in parts)}
    n = c["nx"] * c["ny"] * c["nt"]
    b, f = _step_work(c)
    if kind == "nonlinear":
        return {"bytes": 16 * n, "flops": (5 * 2 * math.log2(c["nt"]) * c["sst"] + (100 if c["plasma"] else 40)) * n}
    if kind == "diag":
        return {"bytes": 8 * n, "flops": (5 * math.log2(c["nt"]) + 12) * n}
    steps = {"fixed": c.get("steps", 1), "adaptive": 3 * c.get("attempts", 1), "ssfm": 1}[kind]
    return {"bytes": 32 * n + steps * b, "flops": steps * f}


# ---- the same in 64 bits --------------------------------------------------------------------------
def _dev(v):
    return torch.from_numpy(np.ascontiguousarray(v)).to("cuda")


def _linear(a, ph, zd, zp):
    """Diffraction over zd (signed) and dispersion over zp, in place of a."""
    f = torch.fft.fftn(a)
    del a
    sh = lambda v: np.roll(v, -(v.size // 2))  # noqa: E731  centred -> FFT order
    for k, axis in (("kx", 2), ("ky", 1)):
        q = _dev(np.exp(-1j * zd * sh(ph[k]) ** 2 / (2 * ph["k0"])))
        f *= q.reshape([-1 if d == axis else 1 for d in range(3)])
    f *= _dev(np.exp(1j * zp * sh(ph["betas"])))[:, None, None]
    return torch.fft.ifftn(f)


def _ions(a, ph):
    """(ions before each slice, sigma, w0 tau sigma) of the ionization model."""
    ip = torch.view_as_real(a).square().sum(-1) * (HBAR * ph["w0"])
    ip[ip == 0] = 1e-30
    e0 = torch.sqrt(2 * ZW0 * ip) * FCTR
    f = e0 / EF
    pot = [ph["i1"] / IH, ph["i2"] / IH]
    kon = ph["dt"] / T0
    rates = []
    for st in range(2):
        nq = (st + 1) / math.sqrt(2 * pot[st])
        k1 = 2.0 ** (2 * nq) / (nq * math.gamma(nq + 1) * math.gamma(nq)) * math.sqrt(6 / math.pi) * pot[st]
        k3 = 2 * (2 * pot[st]) ** 1.5
        w = k1 * torch.pow(k3 / f, 2 * nq - 1.5) * torch.exp(-k3 / (3 * f))
        rates.append(torch.nan_to_num(w, nan=0.0).mul_(kon))
        del w
    del f
    u = e0 * (ph["sig"] * ph["rho_nt"] * EL0 / (math.sqrt(2) * ME * ph["w0"]))
    del e0
    qw = (ph["w0"] ** 2 * (ph["w0"] / C0) / ph["rho_c"]) / (u * u + ph["w0"] ** 2)
    sigma = qw * u / ph["w0"]
    del u
    b = ip * sigma * (kon / ph["i1"])
    del ip
    ions = torch.empty_like(b)
    R, v, s2 = (torch.zeros_like(b[0]) for _ in range(3))
    for t in range(b.shape[0]):
        torch.add(v, s2, alpha=2, out=ions[t])
        R = R + rates[0][t]
        R = R + (1 - R) * b[t]
        new = -torch.expm1(-R) - s2
        s2 = s2 + rates[1][t] * v
        v = new
    return ions, sigma, qw


def _nonlinear(a, ph, dz):
    """a exp(dz A_nl), in place."""
    re = torch.zeros(a.shape, dtype=torch.float64, device=a.device)
    if ph["plasma"]:
        ions, sigma, qw = _ions(a, ph)
        ions *= ph["rho_nt"] / 2
        re = sigma.mul_(ions).neg_()
        im = qw.mul_(ions).neg_()
        del ions, sigma, qw
    else:
        im = torch.zeros_like(re)
    im += ph["gamma2"] * torch.view_as_real(a).square().sum(-1)
    if ph["sst"]:
        w = np.roll(ph["w"], -(ph["nt"] // 2))
        d = torch.fft.fft(a, dim=0)
        d *= _dev(-1j * w)[:, None, None]
        d = torch.fft.ifft(d, dim=0)
        d *= a.conj()
        s = ph["gamma2"] / ph["w0"]
        re -= 3 * s * d.real
        im -= s * d.imag
        del d
    re *= dz
    im *= dz
    a *= torch.polar(re.exp_(), im)
    return a


def _sign(z, lens):
    return 1 if lens else (int(math.floor(z / CAV) + 1) % 2) * 2 - 1


def _fixed64(a, ph, steps, start):
    dz = ph["dz"]
    sign = lambda g: _sign(g * dz + 1e-9 * CAV, ph["lens"])  # noqa: E731
    a = _linear(a, ph, sign(start) * dz / 2, dz / 2)
    for g in range(start, start + steps):
        a = _nonlinear(a, ph, dz)
        crossed = math.floor((g + 1) * dz / CAV + 1e-9) > math.floor(g * dz / CAV + 1e-9)
        last = g == start + steps - 1
        if last or (crossed and ph["lens"]):
            a = _linear(a, ph, sign(g) * dz / 2, dz / 2)
            if crossed and ph["lens"]:
                for k, axis in (("x", 2), ("y", 1)):
                    a *= _dev(np.exp(-1j * ph["k0"] * ph[k] ** 2 / ROC)).reshape([-1 if d == axis else 1 for d in range(3)])
            if not last:
                a = _linear(a, ph, sign(g + 1) * dz / 2, dz / 2)
        else:
            a = _linear(a, ph, (sign(g) + sign(g + 1)) * dz / 2, dz)
    return a


def _adaptive64(a, ph, attempts):
    """Step doubling from z = 0; the attempts stay within the first pass."""
    h, bad = ph["dz"], []
    for _ in range(attempts):
        one = _linear(_nonlinear(_linear(a.clone(), ph, h, h), ph, 2 * h), ph, h, h)
        two = _linear(_nonlinear(_linear(a.clone(), ph, h / 2, h / 2), ph, h), ph, h, h)
        two = _linear(_nonlinear(two, ph, h), ph, h / 2, h / 2)
        err = float(torch.linalg.vector_norm(two - one) / torch.linalg.vector_norm(two))
        if err > 2e-5 and h / 2 > 1e-7:
            h /= 2
            bad.append(1)
            continue
        bad.append(0)
        a = two.mul_(4 / 3).sub_(one, alpha=1 / 3)
        if err > 1e-5:
            h = h / 2 ** (1 / 3) if err < 2e-5 else h
        elif err <= 0.5e-5:
            h *= 2 ** (1 / 3)
    return a, bad, h


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "train":
        return _exact_train(c, seed)
    if kind == "batch":
        if sum(k["nx"] * k["ny"] * k["nt"] for k, _ in _sweep(c, seed)) * c["steps"] > 3e9:
            return None
        out = []
        for k, s in _sweep(c, seed):
            ph = _physics(k)
            a, esig = _field(ph, s)
            out.append(_fixed64(a * math.sqrt(ph["energy"] / esig), ph, c["steps"], 0))
        return {"A": out}
    ph = _physics(c)
    steps = {"fixed": c.get("steps", 0), "adaptive": 3 * c.get("attempts", 0)}.get(kind, 1)
    if c["nx"] * c["ny"] * c["nt"] * steps > 4e9:  # about 20 seconds of 64-bit steps
        return None
    a, esig = _field(ph, seed)
    a *= math.sqrt(ph["energy"] / esig)
    if kind == "fixed":
        return {"A": _fixed64(a, ph, c["steps"], c["from"])}
    if kind == "adaptive":
        a, bad, h = _adaptive64(a, ph, c["attempts"])
        return {"A": a, "bad": np.array(bad), "dz": float(h)}
    if kind == "nonlinear":
        return {"A": _nonlinear(a.to(torch.complex64).to(torch.complex128), ph, ph["dz"])}
    j = HBAR * ph["w0"]
    if kind == "ssfm":
        h = ph["dz"]
        a = _linear(_nonlinear(_linear(a, ph, h / 2, h / 2), ph, h), ph, h / 2, h / 2)
        out = {"A": a.reshape(-1)}
        if c["change"]:
            e = torch.view_as_real(a).square().sum((0, 3)) * (j * ph["dx"] * ph["dt"])
            out.update(BP1=e.sum(0), BP2=e.sum(1))
        return out
    e = torch.view_as_real(a).square().sum(-1)
    out = {"temp": e.sum((1, 2)) * (j * ph["dx"] ** 2), "BP1": e.sum((0, 1)) * (j * ph["dx"] * ph["dt"]),
           "BP2": e.sum((0, 2)) * (j * ph["dx"] * ph["dt"])}
    del e
    f = torch.fft.fft(a, dim=0)
    out["spec"] = torch.view_as_real(f).square().sum((1, 2, 3)) * (j * (ph["dx"] * ph["dt"]) ** 2)
    return out


# ---- the step-size controller's training ----------------------------------------------------------
def _train_data(c, seed):
    """Features on the scales that the propagator's have, and a smooth target (the logarithm of a step length)."""
    r = np.random.default_rng(seed)
    mean = np.array([15, -9, 1, -2, -3, 0.8, 0.0, 0.1, 0.1, -2.5, 0.5, -6, 0.2, -2, 1, 1], dtype=np.float32)
    std = np.array([1, 3, 0.7, 1, 0.4, 0.5, 0.1, 0.03, 0.03, 0.3, 0.3, 0.5, 0.3, 0.5, 0.2, 0.2], dtype=np.float32)
    z = r.standard_normal((c["n"], 16)).astype(np.float32)
    y = (-5 - 0.5 * z[:, 0] + 0.3 * np.sin(z[:, 2]) - 0.2 * z[:, 9] * z[:, 4] + 0.1 * np.abs(z[:, 11])
         + 0.02 * r.standard_normal(c["n"])).astype(np.float32)
    w = (r.uniform(-1, 1, 5313) * np.where(np.arange(5313) < 1088, 0.25, 0.125)).astype(np.float32)
    return z * std + mean, y, mean, std, w


def _prepare_train(c, seed):
    from mpc_gb300 import capi
    X, y, mean, std, w = _train_data(c, seed)
    m = capi.MLP(seed=0)
    m.set_normalization(mean, std, float(y.mean()), float(y.std()))
    return {"c": c, "mlp": m, "X": X, "y": y, "weights": w}


def _shuffles(n, epochs, seed):
    """Fisher-Yates orders driven by splitmix64, one per epoch (each shuffles the one before)."""
    mask, s, p = (1 << 64) - 1, seed, list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            p[i], p[j] = p[j], p[i]
        yield np.array(p)


def _exact_train(c, seed):
    X, y, mean, std, w = _train_data(c, seed)
    f64 = lambda v: torch.from_numpy(np.asarray(v, dtype=np.float64))  # noqa: E731
    xn = (f64(X) - f64(mean)) / f64(std)
    yn = (f64(y) - float(np.float32(y.mean()))) / float(np.float32(y.std()))
    W = f64(w)
    m, v, t, loss = torch.zeros_like(W), torch.zeros_like(W), 0, 0.0
    lr, b1, b2, eps = (float(np.float32(k)) for k in (1e-3, 0.9, 0.999, 1e-8))
    cut = np.cumsum([0, 1024, 64, 4096, 64, 64, 1])
    for order in _shuffles(c["n"], c["epochs"], 7):
        loss = 0.0
        for k in range(0, c["n"], c["batch"]):
            at = torch.from_numpy(order[k:k + c["batch"]])
            q = W.detach().requires_grad_()
            w1, c1, w2, c2, w3, c3 = (q[cut[i]:cut[i + 1]] for i in range(6))
            h = torch.nn.functional.silu(xn[at] @ w1.reshape(64, 16).T + c1)
            h = torch.nn.functional.silu(h @ w2.reshape(64, 64).T + c2)
            e = (h @ w3 + c3 - yn[at]).square().mean()
            (g,) = torch.autograd.grad(e, q)
            loss += float(e) * len(at) / c["n"]
            t += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            W = W - lr * (m / (1 - 0.9**t)) / (torch.sqrt(v / (1 - 0.999**t)) + eps)
    return {"weights": W, "loss": loss}
