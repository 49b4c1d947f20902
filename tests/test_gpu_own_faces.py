"""Meshes small enough that their last kernel forms its elements' face fluxes itself (1D operators, dense operators, mixed
orders), against the CPU oracle: every order, both fluxes, affine and jittered elements, advection, residual and steps (with the limiter), sizes that
leave the last block of elements partly filled, and the side of the line where the fluxes have a kernel of their own.

Tolerance 1e-11 of the largest entry, the repository's FP64 bound."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg
from oracle import Oracle

pytestmark = pytest.mark.gpu

TOL = 1e-11
VORTEX = (2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0)
ADV = dict(pde="advection", num_flux="upwind", test_case="advection_sine", lo=(0, 0, 0), hi=(1, 1, 1), b_adv=(1.0, -0.5, 0.25))
EUL = dict(lo=(-5, -5, 0), hi=(5, 5, 5), vortex=VORTEX)

# (case, kernels per residual)
CASES = {
    "quad-p1": (dict(EUL, d=2, p=1, n_elem=(32, 33, 1)), 2),
    "quad-p2-lf": (dict(EUL, d=2, p=2, n_elem=(12, 11, 1), num_flux="Lax-Friedrichs"), 2),
    "quad-p3-jitter": (dict(EUL, d=2, p=3, n_elem=(19, 17, 1), jitter=0.1, seed=3), 2),
    "quad-p4": (dict(EUL, d=2, p=4, n_elem=(13, 7, 1)), 2),
    "quad-p3-line": (dict(EUL, d=2, p=3, n_elem=(50, 25, 1)), 2),
    "quad-p3-beyond": (dict(EUL, d=2, p=3, n_elem=(51, 25, 1)), 3),
    "hex-p1": (dict(EUL, d=3, p=1, n_elem=(9, 8, 8)), 2),
    "hex-p2-jitter": (dict(EUL, d=3, p=2, n_elem=(5, 4, 3), jitter=0.1, seed=4), 2),
    "hex-p3-lf": (dict(EUL, d=3, p=3, n_elem=(4, 3, 3), num_flux="Lax-Friedrichs"), 2),
    "hex-p4": (dict(EUL, d=3, p=4, n_elem=(3, 3, 2)), 2),
    "dense-quad-p2": (dict(EUL, d=2, p=2, n_elem=(7, 5, 1)), 2),
    "dense-hex-p1-lf": (dict(EUL, d=3, p=1, n_elem=(5, 4, 3), num_flux="Lax-Friedrichs"), 2),
    "tri-p2": (dict(EUL, d=2, element="tri", p=2, n_elem=(33, 33, 1), jitter=0.1, seed=3), 2),
    "tri-p2-beyond": (dict(EUL, d=2, element="tri", p=2, n_elem=(34, 33, 1), jitter=0.1, seed=3), 3),
    "tri-p1to3": (dict(EUL, d=2, element="tri", p=1, p_max=3, p_seed=5, n_elem=(11, 9, 1), jitter=0.1, seed=3), 2),
    "hex-p1to2": (dict(EUL, d=3, p=1, p_max=2, p_seed=5, n_elem=(4, 3, 3), jitter=0.1, seed=3), 2),
    "quad-p2-advection": (dict(ADV, d=2, p=2, n_elem=(13, 11, 1), jitter=0.1, seed=3), 2),
    "hex-p2-advection": (dict(ADV, d=3, p=2, n_elem=(4, 4, 3)), 2),
}


@pytest.mark.parametrize("case,kernels", list(CASES.values()), ids=list(CASES))
def test_residual_and_steps(case, kernels):
    sim = dg.Simulation(dg.Config(**case))
    orc = Oracle(data_model=dg.load_library().dpg_sim_view(sim.handle), threads=8)
    ctx = dg.GpuContext(sim)
    assert dg.load_library().dpg_gpu_launches_per_rhs(ctx.handle) == kernels
    u = sim.sol_coef() * (1.0 + 1e-3 * np.random.default_rng(5).standard_normal(sim.n_dof))
    ctx.upload(u)
    m = ctx.compute_rhs()
    m_ref, r_ref = orc.compute_rhs(u)
    assert np.max(np.abs(ctx.rhs() - r_ref)) <= TOL * np.max(np.abs(r_ref))
    assert abs(m - m_ref) <= TOL * m_ref
    u = sim.sol_coef()
    ctx.upload(u)
    dt = 1e-4
    ctx.rk_step(dt, 3)
    orc.rk_step(u, dt, 3)
    assert np.max(np.abs(ctx.download() - u)) <= TOL * np.max(np.abs(u))
