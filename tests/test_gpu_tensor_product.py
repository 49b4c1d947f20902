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


ANNULUS = dict(d=2, mesh="annulus", lo=(1.0, 0, 0), hi=(2.0, 0, 0), pde="navier_stokes", mu=5e-3, Pr=0.72, omega=0.5,
               test_case="taylor_couette", bc=("noslip_all_rotating", "noslip_adiabatic"))
BOX_NS = dict(d=3, lo=(0, 0, 0), hi=(1, 1, 1), jitter=0.1, seed=4, pde="navier_stokes", mu=1e-2,
              test_case="isentropic_vortex", vortex=(0.5, 0.5, 0.5, 1.0, 0.3, 0.2, 0.1, 1.0),
              bc=("periodic",) * 4 + ("noslip_adiabatic", "noslip_adiabatic"))
SLIP = dict(d=2, lo=(0, 0, 0), hi=(2, 1, 1), test_case="free_stream", vortex=(0, 0, 0, 1.0, 0.7, 0.3, 0, 1.0),
            bc=("riemann", "riemann", "slipwall", "riemann"), bc_state=(1.0, 0.7, 0.3, 0.0, 1.0))

GENERAL = {
    "annulus-p1": dict(ANNULUS, p=1, n_elem=(9, 31, 1)),
    "annulus-p2-lf": dict(ANNULUS, p=2, n_elem=(61, 151, 1), num_flux="Lax-Friedrichs"),   # 28 elements a block, last partial
    "annulus-p3": dict(ANNULUS, p=3, n_elem=(5, 13, 1)),
    "annulus-p4": dict(ANNULUS, p=4, n_elem=(7, 15, 1)),
    "hex-ns-p1": dict(BOX_NS, p=1, n_elem=(5, 4, 3)),
    "hex-ns-p3": dict(BOX_NS, p=3, n_elem=(3, 2, 3)),
    "hex-slip-p4": dict(d=3, p=4, n_elem=(3, 2, 2), lo=(0, 0, 0), hi=(1, 1, 1), jitter=0.1, seed=2, test_case="free_stream",
                        vortex=(0, 0, 0, 1.0, 0.0, 0.3, 0.2, 1.0), bc=("slipwall", "slipwall") + ("periodic",) * 4),
    "slip-p4-affine": dict(SLIP, p=4, n_elem=(7, 5, 1)),
}


@pytest.mark.parametrize("case", list(GENERAL.values()), ids=list(GENERAL))
def test_walls_and_viscous_terms(case):
    """Residual at 1e-11 and Jacobian products at 4e-13 (the reference's linearisation bound) of meshes with boundary
    faces and BR2 terms."""
    sim = dg.Simulation(dg.Config(**case))
    orc = Oracle(sim, threads=8)
    ctx = dg.GpuContext(sim)
    rng = np.random.default_rng(11)
    u0 = orc.initial_solution()
    u = u0 + 1e-2 * np.max(np.abs(u0)) * rng.standard_normal(u0.shape)
    ctx.upload(u)
    m = ctx.compute_rhs()
    m_ref, r_ref = orc.compute_rhs(u)
    assert np.max(np.abs(ctx.rhs() - r_ref)) <= TOL * np.max(np.abs(r_ref))
    assert abs(m - m_ref) <= TOL * m_ref
    v = rng.standard_normal(u.shape)
    cs, _ = orc.jvp_complex_step(u, v)
    assert np.max(np.abs(ctx.jacobian_apply(v) - cs)) <= 4e-13 * np.max(np.abs(cs))


def _advection_rhs(sim, u, b):
    """m_inv rhs by the dense operators; a boundary state is the interior trace."""
    from tests_support import sim_arrays
    a = sim_arrays(sim)
    d, n_fc, nf = a["d"], sim.n_fc, sim.n_face
    u = u.reshape(sim.n_vol, -1)
    s, met = u @ a["cv0_vs_vc"].T, a["metrics_vc"]
    out = sum((sum(met[:, x + d * r] * b[x] for x in range(d)) * s) @ a["tw1_vt_vc"][r].T for r in range(d))
    tr = (u @ a["cv0_vs_fc"].T).reshape(sim.n_vol, a["n_fl"], n_fc)
    side = np.zeros((nf, 2), int) - 1
    for e in range(sim.n_vol):
        for lf in range(a["n_fl"]):
            side[a["vol_face"][e, lf], a["vol_face_side"][e, lf]] = e * a["n_fl"] + lf
    nc, nrm, jf = a["nc_fc"].reshape(nf, n_fc), a["normals_fc"].reshape(nf, n_fc, d), a["jacobian_det_fc"].reshape(nf, n_fc)
    tr = tr.reshape(-1, n_fc)
    for f in range(nf):
        L = tr[side[f, 0]]
        R = tr[side[f, 1]][nc[f]] if side[f, 1] >= 0 else L
        bn = nrm[f] @ np.array(b[:d])
        F = np.where(bn > 2.220446049250313e-16, bn * L, bn * R) * jf[f]
        e, lf = divmod(side[f, 0], a["n_fl"])
        out[e] -= a["tw0_vt_fc"][lf] @ F
        if side[f, 1] >= 0:
            e, lf = divmod(side[f, 1], a["n_fl"])
            G = np.empty(n_fc)
            G[nc[f]] = F
            out[e] += a["tw0_vt_fc"][lf] @ G
    w = a["w_vc"] * a["jacobian_det_vc"].reshape(sim.n_vol, -1)
    M = np.einsum("ci,ec,cj->eij", a["cv0_vs_vc"], w, a["cv0_vs_vc"])
    return np.linalg.solve(M, out[..., None]).ravel()


@pytest.mark.parametrize("p", [3, 5], ids=["p3", "p5-dense"])   # 5: above the 1D operators' orders, the dense kernels
def test_advection_with_boundary_faces_from_lists(p):
    from test_reference_lists import _lists
    box = dg.Simulation(dg.Config(d=2, p=p, n_elem=(4, 3, 1), lo=(0, 0, 0), hi=(1, 1, 1), jitter=0.1, seed=3,
                                  bc=("riemann",) * 4))
    b = (1.0, 0.5, 0.0)
    cfg = dg.Config(d=2, p=p, n_elem=(4, 3, 1), lo=(0, 0, 0), hi=(0, 0, 0), pde="advection", num_flux="upwind",
                    test_case="advection_sine", b_adv=b)
    sim = dg.Simulation.from_reference_lists(cfg, *_lists(box))
    ctx = dg.GpuContext(sim)
    u = sim.sol_coef() + 0.1 * np.random.default_rng(1).standard_normal(sim.n_dof)
    ctx.upload(u)
    ctx.compute_rhs()
    ref = _advection_rhs(sim, u, b)
    assert np.max(np.abs(ctx.rhs() - ref)) <= TOL * np.max(np.abs(ref))
    v = np.random.default_rng(2).standard_normal(sim.n_dof)
    jv = _advection_rhs(sim, v, b)                   # linear
    assert np.max(np.abs(ctx.jacobian_apply(v) - jv)) <= TOL * np.max(np.abs(jv))
