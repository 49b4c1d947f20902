"""The FP64 residual of simplex meshes with its dense products on the tensor cores (meshes above the work threshold) against
the CPU oracle: every order, an order per element, partly filled blocks (25 TETs / 32 TRIs of Euler), both fluxes, steps
with the positivity limiter, scaled states and states that are not finite.

Tolerance 1e-11 of the largest entry, the repository's FP64 bound: the products' own error is below 2^-61 K of the largest
product (K <= 448), the rest is FP64."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg
from oracle import Oracle

pytestmark = pytest.mark.gpu

TOL = 1e-11
TET = dict(d=3, element="tet", jitter=0.1, seed=2, lo=(-5, -5, 0), hi=(5, 5, 2.5), vortex=(2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0))
TRI = dict(d=2, element="tri", jitter=0.1, seed=3, vortex=(2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0))

CASES = {
    "tet-p1": dict(TET, p=1, n_elem=(24, 24, 24)),
    "tet-p2": dict(TET, p=2, n_elem=(13, 12, 11)),
    "tet-p3-lf": dict(TET, p=3, n_elem=(9, 8, 8), num_flux="Lax-Friedrichs"),
    "tet-p4": dict(TET, p=4, n_elem=(8, 6, 5)),
    "tet-p1to4": dict(TET, p=1, p_max=4, p_seed=3, n_elem=(8, 8, 8)),
    "tet-p2to3": dict(TET, p=2, p_max=3, p_seed=5, n_elem=(9, 8, 8)),
    "tri-p2": dict(TRI, p=2, n_elem=(123, 97, 1)),
    "tri-p4": dict(TRI, p=4, n_elem=(65, 61, 1)),
    "tri-p1to4": dict(TRI, p=1, p_max=4, p_seed=5, n_elem=(90, 77, 1)),
}


def _problem(case):
    sim = dg.Simulation(dg.Config(**case))
    orc = Oracle(data_model=dg.load_library().dpg_sim_view(sim.handle), threads=8)
    return sim, orc, dg.GpuContext(sim)


@pytest.mark.parametrize("case", list(CASES.values()), ids=list(CASES))
def test_residual_and_steps(case):
    sim, orc, ctx = _problem(case)
    u = sim.sol_coef() * (1.0 + 1e-3 * np.random.default_rng(5).standard_normal(sim.n_dof))
    ctx.upload(u)
    m = ctx.compute_rhs()
    m_ref, r_ref = orc.compute_rhs(u)
    assert np.max(np.abs(ctx.rhs() - r_ref)) <= TOL * np.max(np.abs(r_ref))
    assert abs(m - m_ref) <= TOL * m_ref
    u = sim.sol_coef()
    ctx.upload(u)
    dt = 1e-4
    ctx.rk_step(dt, 2)
    orc.rk_step(u, dt, 2)
    assert np.max(np.abs(ctx.download() - u)) <= TOL * np.max(np.abs(u))


def test_scaled_state_scales_the_residual():
    """The fluxes are homogeneous of degree 1: a state times 2^k (far from unit magnitudes) gives the residual times 2^k."""
    sim, _, ctx = _problem(CASES["tet-p2"])
    u = sim.sol_coef()
    ctx.upload(u)
    ctx.compute_rhs()
    r = ctx.rhs()
    for k in (-200, 200):
        ctx.upload(np.ldexp(u, k))
        ctx.compute_rhs()
        assert np.max(np.abs(np.ldexp(ctx.rhs(), -k) - r)) <= 1e-13 * np.max(np.abs(r))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_state_is_reported(bad):
    sim, _, ctx = _problem(CASES["tet-p3-lf"])
    u = sim.sol_coef()
    u[sim.n_dof // 2] = bad
    ctx.upload(u)
    with pytest.raises(dg.DpgError) as ei:
        ctx.compute_rhs()
    assert ei.value.status == dg.api.DPG_ERR_NONFINITE
