"""The dense positivity limiter over groups of volumes of one order (one launch for all groups, 32 volumes per block) against
the numpy restatement, on states with a negative density or pressure planted in every fifth volume.  Sizes leave
every group's last block partly filled; the HEX case has n_s = 64, the largest.

Tolerances as for the tensor-product limiter: corrected volumes 1e-10 of the state's largest entry; the others are left bit
identical."""
import ctypes as C

import numpy as np
import pytest

import dpgsolver_gb300 as dg
from positivity_support import EPS_PHYS, bezier_prim_min, limit_volume
from tests_support import DpgSim

pytestmark = pytest.mark.gpu

VORTEX = (2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0)
CASES = {
    "tri-p1": dict(d=2, element="tri", p=1, n_elem=(9, 7, 1)),
    "tet-p4": dict(d=3, element="tet", p=4, n_elem=(4, 3, 3)),
    "tri-p1to4": dict(d=2, element="tri", p=1, p_max=4, p_seed=5, n_elem=(19, 9, 1)),
    "tet-p1to4": dict(d=3, element="tet", p=1, p_max=4, p_seed=5, n_elem=(4, 4, 3)),
    "quad-p1to4": dict(d=2, p=1, p_max=4, p_seed=5, n_elem=(9, 7, 1)),
    "hex-p1to3": dict(d=3, p=1, p_max=3, p_seed=5, n_elem=(5, 4, 3)),
}


@pytest.mark.parametrize("case", list(CASES.values()), ids=list(CASES))
def test_limiter(case):
    sim = dg.Simulation(dg.Config(lo=(-5, -5, 0), hi=(5, 5, 2.5), jitter=0.1, seed=3, vortex=VORTEX, **case))
    s = C.cast(sim.handle, C.POINTER(DpgSim)).contents
    d, nv = s.d, s.n_var
    rng = np.random.default_rng(1)
    u = np.array(sim.sol_coef())
    rows = []
    for e in range(s.n_vol):
        o = s.ops[s.vol_ops[e]]
        ub = u[s.vol_dof_off[e]:s.vol_dof_off[e + 1]].reshape(nv, o.n_s)
        rows.append((ub, o))
        if e % 5:
            continue
        if e % 2:
            m2 = np.sum(ub[1:1 + d, 0] ** 2)
            ub[d + 1, 0] = 0.5 * m2 / ub[0, 0] * (1.0 - rng.uniform(0.25, 0.75))
        else:
            ub[0, 0] = -rng.uniform(0.01, 0.05)
    ctx = dg.GpuContext(sim)
    ctx.upload(u)
    ctx.enforce_positivity()
    g, scale = ctx.download(), np.max(np.abs(u))
    for e, (ub, o) in enumerate(rows):
        ge = g[s.vol_dof_off[e]:s.vol_dof_off[e + 1]].reshape(nv, o.n_s)
        sb = np.ctypeslib.as_array(o.ccSB0_vs_vs, shape=(o.n_s, o.n_s))
        bs = np.ctypeslib.as_array(o.ccBS0_vs_vs, shape=(o.n_s, o.n_s))
        if min(bezier_prim_min(ub, sb, d)) < EPS_PHYS:   # planted, or a coarse interpolant that needs it
            ref, ok = limit_volume(ub, sb, bs, d)
            assert ok
            assert np.max(np.abs(ge - ref)) <= 1e-10 * scale
        else:
            assert e % 5
            assert np.array_equal(ge, ub)
