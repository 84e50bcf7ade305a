"""The bounded grid barrier of the cooperative kernels (csrc/coop.cuh): a wait that
runs out leaves the kernel's status unwritten.  tests/cuda/coop_check.cu, built with
nvcc for sm_103a and run on the GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_reported(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "coop_check")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                        "-I", os.path.join(ROOT, "topopt_in_petsc_transient_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cuda", "coop_check.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "barrier OK" in r.stdout, r.stdout + r.stderr
