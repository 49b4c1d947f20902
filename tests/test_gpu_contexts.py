"""Two live contexts whose kernels are the same functions with different amounts of shared memory: the second one's set-up leaves
the first one's launches as they were.  The residual is repeated bit for bit and the steps run."""
import numpy as np
import pytest

import dpgsolver_gb300 as dg

pytestmark = pytest.mark.gpu

VORTEX = (2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0)
EUL = dict(lo=(-5, -5, 0), hi=(5, 5, 5), vortex=VORTEX)
ADV = dict(pde="advection", num_flux="upwind", test_case="advection_sine", lo=(0, 0, 0), hi=(1, 1, 1), b_adv=(1.0, -0.5, 0.25),
           jitter=0.1, seed=3)
HEX = dict(EUL, d=3, p=1, p_max=3, p_seed=5, jitter=0.1, seed=3)

PAIRS = {
    "hex-p1to3-fine-coarse": (dict(HEX, n_elem=(24, 16, 8)), dict(HEX, n_elem=(4, 4, 4)), 0),
    "advection-tet-p2-tri-p1": (dict(ADV, d=3, element="tet", p=2, n_elem=(4, 3, 3)), dict(ADV, d=2, element="tri", p=1, n_elem=(5, 4, 1)), 0),
    "advection-tet-p4-tet-p1": (dict(ADV, d=3, element="tet", p=4, n_elem=(4, 3, 3)), dict(ADV, d=3, element="tet", p=1, n_elem=(3, 3, 3)), 0),
    "advection-quad-p1to4": (dict(ADV, d=2, p=1, p_max=4, p_seed=5, n_elem=(20, 20, 1)), dict(ADV, d=2, p=1, p_max=2, p_seed=5, n_elem=(3, 3, 1)), 0),
    "split-hex-p2-tet-p3": (dict(EUL, d=3, p=2, n_elem=(6, 5, 4)), dict(EUL, d=3, element="tet", p=3, n_elem=(3, 3, 3)), 7),
    "split-quad-p4-tri-p1": (dict(EUL, d=2, p=4, n_elem=(9, 8, 1)), dict(EUL, d=2, element="tri", p=1, n_elem=(4, 4, 1)), 7),
}


@pytest.mark.parametrize("first,second,split", list(PAIRS.values()), ids=list(PAIRS))
def test_second_context_leaves_the_first_one_running(first, second, split):
    def context(case):
        ctx = dg.GpuContext(dg.Simulation(dg.Config(**case)))
        if split:
            ctx.set_precision(dg.PREC_BF16_SLICED, split)
        return ctx

    a = context(first)
    m = a.compute_rhs()
    r = a.rhs()
    b = context(second)
    b.compute_rhs()
    assert a.compute_rhs() == m
    assert np.array_equal(a.rhs(), r)
    b.rk_step(1e-4, 2)
    a.rk_step(1e-4, 2)
    assert np.all(np.isfinite(a.download())) and np.all(np.isfinite(b.download()))
