"""The control of the PDE filter's solve (csrc/filtctl.cuh) on the host:
tests/cuda/filter_control_check.cu steps the solve in the kernel's arithmetic with
the kernel's own scalars, for fields and radii from the usual ones to those that
FP32 cannot represent, and checks that every solve ends and that what CG in FP64
alone solves is solved."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_solve_ends_as_fp64_alone_would(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "filter_control_check")
    r = subprocess.run([nvcc, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "topopt_in_petsc_transient_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cuda", "filter_control_check.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "control OK" in r.stdout, r.stdout + r.stderr
