"""Which kernels an FP64 residual launches (recorded with torch's profiler): the form that the set-up's rules pick, on both sides
of their lines.  The accuracy of each form is tested elsewhere; here a test that means to cover one cannot pass on another."""
import pytest

import dpgsolver_gb300 as dg

pytestmark = pytest.mark.gpu

EUL = dict(lo=(-5, -5, 0), hi=(5, 5, 2.5), vortex=(2.5, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0))
TET = dict(EUL, d=3, element="tet", jitter=0.1, seed=2)
TRI = dict(EUL, d=2, element="tri", jitter=0.1, seed=3)
ADV = dict(pde="advection", num_flux="upwind", test_case="advection_sine", lo=(0, 0, 0), hi=(1, 1, 1), b_adv=(1.0, -0.5, 0.25),
           jitter=0.1, seed=3)
SLICED, DENSE, MIXED, TENSOR = {"k_oz_interp", "k_oz_flux", "k_oz_lift"}, {"k_trace", "k_volume"}, {"k_hp_trace", "k_hp_volume"}, {"k_tp_volume", "k_tp_lift"}

# (case, kernels): the simplex cases of test_gpu_oz.py and both sides of its line, mixed orders, advection, 1D operators
CASES = {
    "tet-p1": (dict(TET, p=1, n_elem=(24, 24, 24)), DENSE | {"k_face"}),     # 800 multiply-adds a volume
    "tet-p2": (dict(TET, p=2, n_elem=(13, 12, 11)), SLICED),
    "tet-p2-small": (dict(TET, p=2, n_elem=(4, 4, 4)), DENSE),
    "tet-p3-lf": (dict(TET, p=3, n_elem=(9, 8, 8), num_flux="Lax-Friedrichs"), SLICED),
    "tet-p4": (dict(TET, p=4, n_elem=(8, 6, 5)), SLICED),
    "tet-p1to4": (dict(TET, p=1, p_max=4, p_seed=3, n_elem=(8, 8, 8)), SLICED),
    "tet-p2to3": (dict(TET, p=2, p_max=3, p_seed=5, n_elem=(9, 8, 8)), SLICED),
    "tri-p2": (dict(TRI, p=2, n_elem=(123, 97, 1)), DENSE | {"k_face"}),     # 864
    "tri-p3": (dict(TRI, p=3, n_elem=(64, 60, 1)), DENSE | {"k_face"}),      # 2,400
    "tri-p4": (dict(TRI, p=4, n_elem=(65, 61, 1)), SLICED),
    "tri-p1to4": (dict(TRI, p=1, p_max=4, p_seed=5, n_elem=(90, 77, 1)), SLICED),
    "tri-p1to3": (dict(TRI, p=1, p_max=3, p_seed=5, n_elem=(40, 40, 1)), MIXED | {"k_hp_face"}),
    "tri-p3-advection": (dict(ADV, d=2, element="tri", p=3, n_elem=(12, 11, 1)), {"k_hp_trace", "k_hp_advect"}),
    "quad-p2": (dict(EUL, d=2, p=2, n_elem=(60, 60, 1)), TENSOR | {"k_face"}),
    "quad-p2-own-faces": (dict(EUL, d=2, p=2, n_elem=(12, 12, 1)), TENSOR),
    "quad-p2-small": (dict(EUL, d=2, p=2, n_elem=(8, 8, 1)), DENSE),
}


def _kernels(run):
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    names = set()
    for _ in range(3):   # a process' first profile may record nothing, or not from its start
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(3):
                run()
            torch.cuda.synchronize()
        for e in prof.events():
            names |= {part for part in e.name.replace("<", " ").replace("(", " ").replace("::", " ").split() if part.startswith("k_")}
        if names:
            return names
    pytest.skip("the profiler records no kernels here")


@pytest.mark.parametrize("case,kernels", list(CASES.values()), ids=list(CASES))
def test_form_of_the_residual(case, kernels):
    ctx = dg.GpuContext(dg.Simulation(dg.Config(**case)))
    ctx.compute_rhs()
    assert _kernels(ctx.compute_rhs) == kernels
