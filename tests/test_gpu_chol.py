"""The panelled Cholesky factorisation of the coarsest operator
(csrc/kernels.cuh): the blocks of a panel give the same factor in any order, and
A times the inverse is the identity.  tests/cuda/chol_check.cu, built with nvcc
for sm_103a and run on the GPU; orders below, at and above a panel of 32."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_panels_in_any_order(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "chol_check")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                        "-I", os.path.join(ROOT, "topopt_in_petsc_transient_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cuda", "chol_check.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "cholesky OK" in r.stdout, r.stdout + r.stderr
