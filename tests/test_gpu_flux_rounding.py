"""Rounding of the FP64 numerical fluxes that large meshes take (numflux_.._rs): no larger than that of the plain formulas.

Tolerance: 1.15 times the plain form's rms error per component and regime (flux_rounding.cu)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_rms_error_of_the_fluxes():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out_dir = os.path.join(HERE, "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "flux_rounding")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + os.path.join(ROOT, "dpgsolver_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(HERE, "flux_rounding.cu")], check=True)
    proc = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(proc.stdout)
    assert proc.returncode == 0, proc.stdout + proc.stderr
    assert "all checks passed" in proc.stdout
