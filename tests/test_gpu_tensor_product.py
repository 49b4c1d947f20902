"""The one-direction-at-a-time operators of the FP64 form (QUAD / HEX, p = 1..4) against the CPU oracle's dense ones:
every order, blocks filled with as many elements as fit and a partly filled last one, single elements, affine and jittered
meshes.  Tolerance: the FP64 parity bound of the repository's residual tests, 1e-11 of the largest entry (sums of at most
5 terms per direction against the dense sums of up to n_c d + n_fc n_fl terms); tangents: the same bound against the
oracle's complex-step products."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg
from oracle import Oracle

pytestmark = pytest.mark.gpu

TOL = 1e-11

CASES = [
    dict(d=2, p=1, n_elem=(160, 122, 1)),                        # 64 elements a block, the last block one short of full
    dict(d=2, p=2, n_elem=(97, 89, 1)),                          # 28 elements a block, 8,633 = 28 x 308 + 9
    dict(d=2, p=3, n_elem=(71, 69, 1), jitter=0.15, seed=3),     # 16 elements a block, per-node metrics
    dict(d=2, p=4, n_elem=(61, 51, 1), num_flux="Lax-Friedrichs"),
    dict(d=3, p=1, n_elem=(23, 22, 20)),                         # 32 elements a block
    dict(d=3, p=2, n_elem=(15, 14, 13), jitter=0.1, seed=4),
    dict(d=3, p=3, n_elem=(11, 11, 11)),
    dict(d=3, p=4, n_elem=(9, 9, 8), num_flux="Lax-Friedrichs"), # 2 elements of 125 threads
    dict(d=3, p=4, n_elem=(3, 3, 3), jitter=0.1, seed=5),        # one element a block
    dict(d=3, p=3, n_elem=(9, 8, 7), pde="advection", num_flux="upwind", test_case="advection_sine", lo=(0, 0, 0),
         hi=(1, 1, 1), b_adv=(1.0, 0.5, 0.25)),
]


def _id(c):
    return f"{c['d']}d-p{c['p']}-{'x'.join(map(str, c['n_elem']))}{'-jitter' if c.get('jitter') else ''}-{c.get('pde', 'euler')}"


@pytest.mark.parametrize("case", CASES, ids=_id)
def test_residual_matches_oracle(case):
    sim = dg.Simulation(dg.Config(**case))
    orc = Oracle(sim, threads=8)
    ctx = dg.GpuContext(sim)
    sol = sim.sol_coef() * (1.0 + 1e-2 * np.random.default_rng(7).standard_normal(sim.n_dof))
    ctx.upload(sol)
    m = ctx.compute_rhs()
    m_ref, r_ref = orc.compute_rhs(sol)
    assert np.max(np.abs(ctx.rhs() - r_ref)) <= TOL * np.max(np.abs(r_ref))
    assert abs(m - m_ref) <= TOL * m_ref


@pytest.mark.parametrize("case", [CASES[2], CASES[5], CASES[8]], ids=_id)
def test_steps_match_oracle(case):
    sim = dg.Simulation(dg.Config(**case))
    orc = Oracle(sim, threads=8)
    ctx = dg.GpuContext(sim)
    sol = sim.sol_coef()
    dt = 0.25 * sim.cfl_dt(0.4, 10.0 / max(case["n_elem"]))
    ctx.rk_step(dt, 2)
    ref = sol.copy()
    orc.rk_step(ref, dt, 2)
    assert np.max(np.abs(ctx.download() - ref)) <= TOL * np.max(np.abs(ref))
