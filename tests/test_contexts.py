"""Contexts of this library made after a device reset and in a second CUDA context of the same device: the
kernels' attributes belong to the CUDA context, so each mpc_create has to set them.  Run in a child process,
whose own primary context is the one that is reset."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, sys
import numpy as np
from mpc_gb300 import inputs
from mpc_gb300.capi import Propagator, load

n, nt, variant, how = int(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3]), sys.argv[4]
p, A = inputs.make_cell(inputs.cell64(Nx=n, Ny=n, Nt=nt))

def run():
    with Propagator(p.copy(variant=variant)) as prop:
        prop.upload(A, calibrate=True)
        prop.run_fixed(3)
        prop.step_double()
        prop.diag()
        return prop.download()

load()
first = run()
if how == "reset":
    rt = C.CDLL("libcudart.so.13")          # the runtime that the library itself is linked to
    assert rt.cudaDeviceReset() == 0        # ends this process's own context, nothing else
    assert np.array_equal(run(), first)
else:
    cu = C.CDLL("libcuda.so.1")
    ctx, back = C.c_void_p(), C.c_void_p()
    assert cu.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0      # made current
    assert np.array_equal(run(), first)
    assert cu.cuCtxPopCurrent_v2(C.byref(back)) == 0 and back.value == ctx.value
    assert cu.cuCtxDestroy_v2(ctx) == 0
    assert np.array_equal(run(), first)                    # the primary context again
print("contexts ok")
"""


@pytest.mark.parametrize("how", ["reset", "second"])
@pytest.mark.parametrize("n,nt,variant", [(16, 64, 0), (64, 512, 2), (128, 1024, 0), (128, 1024, 5)])
def test_new_cuda_context(gpu_lib, n, nt, variant, how):
    r = subprocess.run([sys.executable, "-c", CHILD, str(n), str(nt), str(variant), how], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "contexts ok" in r.stdout, r.stdout + r.stderr
