"""What is said about a variant's plane passes: bench.py's bytes per sweep and mpc_run's line."""
import importlib.util
import os
import subprocess

import pytest

from mpc_gb300 import build, inputs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bench_counts_the_passes_of_each_plane_form():
    spec = importlib.util.spec_from_file_location("bench_passes", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    assert [bench.sweep_passes("plane", {"PL": k}) for k in range(1, 6)] == [1, 2, 2, 2, 1]
    assert [bench.sweep_passes("pencil", {"PL": k}) for k in range(1, 6)] == [1] * 5


@pytest.mark.gpu
@pytest.mark.parametrize("variant,text", [(0, "plane cluster"), (2, "whole planes in shared memory, one pass")])
def test_driver_names_the_plane_passes(gpu_lib, tmp_path, variant, text):
    d = str(tmp_path / "data")
    inputs.write_run(inputs.cell64(cav=0.05, passes=1, steps_per_pass=4), d, nrun=1)
    r = subprocess.run([build.build_driver(), "-d", d, "-n", "1", "-f", "4", "-v", str(variant)], cwd=tmp_path, capture_output=True,
                       text=True)
    assert r.returncode == 0 and text in r.stdout and f"Kernel variant {variant} " in r.stdout, r.stdout + r.stderr
