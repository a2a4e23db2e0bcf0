"""The exit pass's integer conversion (mpc_scale.h, compiled for the host) has the bits of the FP64
multiplication, for every exponent of the FP32 value."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "mpc_scale.h"
extern "C" void scaled(const float* a, double scale, double* out, long n) {
    const mpc::IntScale s = mpc::int_scale(scale);
    for (long i = 0; i < n; i++) out[i] = mpc::scaled_double(a[i], scale, s);
}
extern "C" int is_fast(double scale) { return mpc::int_scale(scale).nexp != 0; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("scale")
    (d / "s.cpp").write_text(SRC)
    so = str(d / "libscale.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mpc_gb300", "csrc"),
                    str(d / "s.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.scaled.argtypes = [C.c_void_p, C.c_double, C.c_void_p, C.c_long]
    lib.is_fast.argtypes = [C.c_double]
    return lib


def _values():
    """Every sign and exponent (zeros, denormals, infinities and NaN with them), mantissas at both ends and
    at random."""
    rng = np.random.default_rng(7)
    man = np.concatenate([[0, 1, 2, 3, 0x400000, 0x7ffffe, 0x7fffff], rng.integers(0, 1 << 23, 500)]).astype(np.uint32)
    e = np.arange(256, dtype=np.uint32)
    bits = (e[:, None] << 23 | man[None, :]).reshape(-1)
    return np.concatenate([bits, bits | np.uint32(0x80000000)]).view(np.float32)


@pytest.mark.parametrize("scale", [
    1.0, 2.0, 0.5, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), np.nextafter(1.0, 0.0), 1.5, 1.0 / 3.0, np.pi,
    9.76e16, 3.1e-7, 1e-30, 1e30, 2.0 ** 895 * 0.99, 2.0 ** -896, 2.0 ** -896 * 0.9, 2.0 ** 1000, 1e-310, 0.0, -1.25, np.inf,
    1.0 + 2.0 ** -24, 1.0 + 2.0 ** -29, 4503599627370497.0 / 2 ** 52, 6004799503160661.0 / 2 ** 52])
def test_bits_of_the_fp64_product(lib, scale):
    a = _values()
    out = np.empty(a.size)
    lib.scaled(a.ctypes.data, float(scale), out.ctypes.data, a.size)
    with np.errstate(all="ignore"):
        ref = a.astype(np.float64) * float(scale)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(out), nan)
    assert np.array_equal(out[~nan].view(np.uint64), ref[~nan].view(np.uint64))


def test_random_factors(lib):
    rng = np.random.default_rng(11)
    a = (rng.standard_normal(20000) * 10.0 ** rng.uniform(-30, 30, 20000)).astype(np.float32)
    out = np.empty(a.size)
    for scale in 10.0 ** rng.uniform(-20, 20, 200):
        lib.scaled(a.ctypes.data, float(scale), out.ctypes.data, a.size)
        assert np.array_equal(out, a.astype(np.float64) * scale)


def test_factors_of_fields_take_the_integer_path(lib):
    for w0 in (1e12, 2.35e15, 1e19):                      # 1 / sqrt(hbar w0 / 1e16)
        assert lib.is_fast(1.0 / np.sqrt(1.054560652926899e-34 * w0 / 1e16))
    assert not lib.is_fast(0.0) and not lib.is_fast(-1.0) and not lib.is_fast(np.inf) and not lib.is_fast(np.nan)
