"""The split precision on a gas at rest: a vortex whose velocity decays to nothing, so that |V|^2 of some face nodes lies below
the smallest normal FP32 number, and the double-float square roots on such operands.

Tolerances: 1e-10 of the largest residual entry, the S = 7 bound against the oracle (test_gpu_split.py); the roots 2^-44
relative, the bound of test_gpu_df64.py."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import dpgsolver_gb300 as dg
from oracle import Oracle

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_roots_of_small_numbers():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out_dir = os.path.join(HERE, "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "df64_small")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + os.path.join(ROOT, "dpgsolver_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(HERE, "df64_small.cu")], check=True)
    proc = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    print(proc.stdout)
    assert proc.returncode == 0, proc.stdout + proc.stderr
    assert "all checks passed" in proc.stdout


# vortex strength, centre, free stream at rest
AT_REST = dict(lo=(-12, -12, 0), hi=(12, 12, 2), vortex=(5.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0))


@pytest.mark.parametrize("flux", ["Lax-Friedrichs", "Roe-Pike"])
@pytest.mark.parametrize("case", [dict(d=2, p=2, n_elem=(37, 31, 1)), dict(d=3, p=1, n_elem=(40, 36, 2)),
                                  dict(d=3, p=2, n_elem=(9, 8, 2), element="tet")], ids=["quad-p2", "hex-p1", "tet-p2"])
def test_vortex_in_a_gas_at_rest(case, flux):
    sim = dg.Simulation(dg.Config(**case, **AT_REST, num_flux=flux))
    u = sim.sol_coef()
    _, ref = Oracle(data_model=dg.load_library().dpg_sim_view(sim.handle), threads=8).compute_rhs(u)
    ctx = dg.GpuContext(sim)
    ctx.set_precision(dg.PREC_BF16_SLICED, 7)
    m = ctx.compute_rhs()
    assert np.max(np.abs(ctx.rhs() - ref)) <= 1e-10 * np.max(np.abs(ref))
    assert abs(m - np.max(np.abs(ref))) <= 1e-10 * np.max(np.abs(ref))
