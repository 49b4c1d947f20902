"""Steady solves on meshes of 1,024 nodes or more (the 1D operators): the residual reaches the rounding level that the forms
before them had.

Navier-Stokes between cylinders, 32x64 QUAD p = 3: the residual at rest is (2.2 +- 0.4)e-11 with dense operators and stored
gradients and with the 1D operators; traces extrapolated from the Gauss points leave it at twice that.  Tolerance 4e-11.
Uniform streams: 1e-11, the tolerance of the periodic Newton solves."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg

pytestmark = pytest.mark.gpu


def test_navier_stokes_annulus_comes_to_rest():
    sim = dg.Simulation(dg.Config(d=2, p=3, n_elem=(32, 64, 1), mesh="annulus", lo=(1.0, 0.0, 0.0), hi=(2.0, 0.0, 0.0),
                                  pde="navier_stokes", mu=5e-3, Pr=0.72, omega=0.5, test_case="taylor_couette",
                                  bc=("noslip_all_rotating", "noslip_adiabatic")))
    ctx = dg.GpuContext(sim)
    st = ctx.newton_solve(dg.PRECOND_BLOCK_ILU, tol=4e-11, cfl_initial=10.0, gmres_restart=200, max_gmres=800, gmres_rtol=1e-4,
                          max_newton=30, ilu_order=dg.api.ILU_ORDER_VOLUME, ilu_parts=8)
    assert st.residual_final <= 4e-11
    assert ctx.compute_rhs() <= 4e-11


@pytest.mark.parametrize("bc", [("periodic",) * 6, ("riemann", "riemann", "slipwall", "slipwall", "periodic", "periodic")],
                         ids=["periodic", "walls"])
def test_uniform_stream_comes_to_rest(bc):
    walls = bc[0] == "riemann"
    v = 0.0 if walls else 0.3
    sim = dg.Simulation(dg.Config(d=2, p=2, n_elem=(14, 12, 1), test_case="free_stream", bc=bc, bc_state=(1.0, 0.6, v, 0.0, 1.0),
                                  vortex=(5.0, 0.0, 0.0, 1.0, 0.6, v, 0.0, 1.0)))
    ctx = dg.GpuContext(sim)
    u = sim.sol_coef()
    r = np.random.default_rng(1).standard_normal((sim.n_vol, sim.n_dof // sim.n_vol))
    ctx.upload(u + (1e-2 * (r - np.roll(r, 1, axis=0))).ravel())
    st = ctx.newton_solve(dg.PRECOND_BLOCK_ILU, tol=1e-11, dtau0=10.0, max_newton=40, gmres_restart=60, max_gmres=600, gmres_rtol=1e-4)
    assert st.residual_final <= 1e-11
