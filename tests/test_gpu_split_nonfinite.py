"""A state that is not finite, and one whose flux is not (negative pressure, Roe-Pike), in the split precisions: the residual is
reported as not finite, as in FP64, and the context goes on with the next state."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg

pytestmark = pytest.mark.gpu

EUL = dict(lo=(-5, -5, 0), hi=(5, 5, 2.5), vortex=(2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0))
CASES = {
    "quad-p3": dict(d=2, p=3, n_elem=(9, 8, 1)),
    "hex-p2": dict(d=3, p=2, n_elem=(12, 11, 3)),
    "hex-p3": dict(d=3, p=3, n_elem=(12, 12, 8)),
    "tet-p2": dict(d=3, p=2, n_elem=(4, 4, 3), element="tet"),
}
MODES = {"sliced7": (dg.PREC_BF16_SLICED, 7), "sliced4": (dg.PREC_BF16_SLICED, 4), "tf32x3": (dg.PREC_TF32X3, 0),
         "bf16x3": (dg.PREC_BF16X3, 0)}


@pytest.mark.parametrize("mode", list(MODES.values()), ids=list(MODES))
@pytest.mark.parametrize("case", list(CASES.values()), ids=list(CASES))
def test_not_finite_is_reported(case, mode):
    sim = dg.Simulation(dg.Config(**case, **EUL))
    ctx = dg.GpuContext(sim)
    u = sim.sol_coef()
    per, n_s = sim.n_dof // sim.n_vol, sim.n_s
    ctx.set_precision(*mode)
    ctx.upload(u)
    ctx.compute_rhs()
    r = ctx.rhs()

    def planted(element, value, variable, node):
        v = u.copy()
        v[element * per + variable * n_s + node] = value
        return v

    bad = [planted(0, np.nan, 0, 0), planted(sim.n_vol - 1, np.inf, sim.n_var - 1, n_s - 1),
           planted(sim.n_vol // 2, -np.inf, 1, n_s // 2)]
    v = u.copy()   # an element of negative pressure
    e = sim.n_vol // 3
    v[e * per + (sim.n_var - 1) * n_s:(e + 1) * per] *= -1.0
    bad.append(v)
    for v in bad:
        ctx.upload(v)
        with pytest.raises(dg.DpgError) as ei:
            ctx.compute_rhs()
        assert ei.value.status == dg.api.DPG_ERR_NONFINITE
    ctx.upload(u)
    ctx.compute_rhs()
    assert np.array_equal(ctx.rhs(), r)
