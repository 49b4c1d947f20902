"""Advection on simplices, where a step is one launch per stage (volume part folded, face fluxes and the next stage's traces
in the same kernel): one order and mixed ones, against the CPU oracle.  Sizes that leave the last block of a group
partly filled, a single block, and p = 4 TETs (operators too large for shared memory).

Tolerance 1e-11 of the largest entry, the repository's FP64 bound."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg
from oracle import Oracle

pytestmark = pytest.mark.gpu

TOL = 1e-11
BASE = dict(pde="advection", num_flux="upwind", test_case="advection_sine", lo=(0, 0, 0), hi=(1, 1, 1), jitter=0.1, seed=3)
TRI = dict(BASE, d=2, element="tri", b_adv=(1.0, -0.5, 0.0))
TET = dict(BASE, d=3, element="tet", b_adv=(1.0, -0.5, 0.25))

CASES = {
    "tri-p1": dict(TRI, p=1, n_elem=(3, 3, 1)),
    "tri-p1-odd": dict(TRI, p=1, n_elem=(23, 17, 1)),
    "tri-p2": dict(TRI, p=2, n_elem=(11, 7, 1)),
    "tri-p3": dict(TRI, p=3, n_elem=(9, 5, 1)),
    "tri-p4": dict(TRI, p=4, n_elem=(13, 5, 1)),
    "tri-p1to4": dict(TRI, p=1, p_max=4, p_seed=5, n_elem=(19, 13, 1)),
    "tet-p1": dict(TET, p=1, n_elem=(3, 3, 3)),
    "tet-p2": dict(TET, p=2, n_elem=(5, 4, 3)),
    "tet-p4": dict(TET, p=4, n_elem=(4, 3, 3)),
    "tet-p1to4": dict(TET, p=1, p_max=4, p_seed=5, n_elem=(5, 4, 3)),
}


@pytest.mark.parametrize("case", list(CASES.values()), ids=list(CASES))
def test_residual_and_steps(case):
    sim = dg.Simulation(dg.Config(**case))
    orc = Oracle(data_model=dg.load_library().dpg_sim_view(sim.handle), threads=4)
    ctx = dg.GpuContext(sim)
    u = sim.sol_coef() * (1.0 + 1e-2 * np.random.default_rng(5).standard_normal(sim.n_dof))
    ctx.upload(u)
    m = ctx.compute_rhs()
    m_ref, r_ref = orc.compute_rhs(u)
    assert np.max(np.abs(ctx.rhs() - r_ref)) <= TOL * np.max(np.abs(r_ref))
    assert abs(m - m_ref) <= TOL * m_ref
    dt = 1e-3
    m = ctx.rk_step(dt, 3)
    m_ref = orc.rk_step(u, dt, 3)
    assert np.max(np.abs(ctx.download() - u)) <= TOL * np.max(np.abs(u))
    if m is not None and m_ref is not None:
        assert abs(m - m_ref) <= TOL * m_ref
