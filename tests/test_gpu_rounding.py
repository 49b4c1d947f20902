"""Rounding of the FP64 residual with the 1D operators (QUAD, HEX): against the same residual in extended precision (numpy
long double: 64 or 113 bits), no larger than that of the dense kernels, which dpg_gpu_compute_rhs_noalloc runs.

The boxes have vertices and element sizes that are FP64 numbers, so that the geometry rounds nothing in either form; the state
is a vortex with 1e-3 of noise.  Tolerance: 1.1 times the dense kernels' rms error (the sampling error of an rms over the
10,000 entries or more is 1 %)."""
import ctypes as C

import numpy as np
import pytest

import dpgsolver_gb300 as dg
from test_zz_no_alloc import _device_mesh, _entry

pytestmark = pytest.mark.gpu

L = np.longdouble


def _legendre(n, x):
    """P_n and its derivative."""
    p0, p1 = np.ones_like(x), x
    for k in range(1, n):
        p0, p1 = p1, ((2 * k + 1) * x * p1 - k * p0) / L(k + 1)
    return (p1, n * (p0 - x * p1) / (1 - x * x)) if n else (p0, 0 * x)


def _gauss(n):
    x = np.polynomial.legendre.leggauss(n)[0].astype(L)
    for _ in range(3):
        p, dp = _legendre(n, x)
        x = x - p / dp
    _, dp = _legendre(n, x)
    return x, 2 / ((1 - x * x) * dp * dp)


def _lobatto(n):
    x = np.sort(np.real(np.polynomial.legendre.Legendre.basis(n - 1).deriv().roots())).astype(L)
    for _ in range(3 if n > 2 else 0):   # (1 - x^2) P'' = 2 x P' - m (m + 1) P
        p, dp = _legendre(n - 1, x)
        x = x - dp * (1 - x * x) / (2 * x * dp - n * (n - 1) * p)
    return np.concatenate([[L(-1)], x, [L(1)]])


def _lagrange(nodes, x):
    """Values and derivatives [len(x), len(nodes)] of the Lagrange polynomials on the nodes."""
    n = len(nodes)
    v, d = np.ones((len(x), n), L), np.zeros((len(x), n), L)
    for i in range(n):
        for j in range(n):
            if j != i:
                v[:, i] *= (x - nodes[j]) / (nodes[i] - nodes[j])
        for k in range(n):
            if k != i:
                t = np.full(len(x), 1 / (nodes[i] - nodes[k]))
                for j in range(n):
                    if j not in (i, k):
                        t = t * (x - nodes[j]) / (nodes[i] - nodes[j])
                d[:, i] += t
    return v, d


def _along(M, x, a):
    """M applied along direction a (the last axis is direction 0)."""
    x = np.moveaxis(x, -1 - a, -1)
    return np.moveaxis((x[..., None, :] * M).sum(-1), -1, -1 - a)


def _flux(s, d, r):
    """Euler flux along axis r of the states s [element, variable, ..]; velocities, pressure."""
    vel = [s[:, 1 + a] / s[:, 0] for a in range(d)]
    p = L(0.4) * (s[:, d + 1] - s[:, 0] * sum(v * v for v in vel) / 2)
    f = [s[:, 1 + r]] + [s[:, 1 + a] * vel[r] + (p if a == r else 0) for a in range(d)] + [(s[:, d + 1] + p) * vel[r]]
    return np.stack(f, axis=1), vel, p


def _numflux(W, R, d, r, kind, sgn):
    """Numerical flux along + axis r of the states below (W) and above (R); sgn -1: the upper element is the face's left
    one and the normal points down (the entropy fix of Roe-Pike is not symmetric)."""
    low = sgn < 0
    W, R = np.where(low, R, W), np.where(low, W, R)
    sgn = sgn[:, 0]   # [element, node ..]
    fl, vl, pl = _flux(W, d, r)
    fr, vr, pr = _flux(R, d, r)
    if kind == "Lax-Friedrichs":
        m = np.maximum(np.sqrt(sum(v * v for v in vl)) + np.sqrt(L(1.4) * pl / W[:, 0]),
                       np.sqrt(sum(v * v for v in vr)) + np.sqrt(L(1.4) * pr / R[:, 0]))
        return (fl + fr + (sgn * m)[:, None] * (W - R)) / 2
    q = np.sqrt(R[:, 0] / W[:, 0])
    u = [(a + q * b) / (1 + q) for a, b in zip(vl, vr)]
    H = ((W[:, d + 1] + pl) / W[:, 0] + q * (R[:, d + 1] + pr) / R[:, 0]) / (1 + q)
    rho, c = q * W[:, 0], np.sqrt(L(0.4) * (H - sum(v * v for v in u) / 2))
    nl, nr, nu = sgn * vl[r], sgn * vr[r], sgn * u[r]
    l1 = np.minimum(np.abs(nl - c), np.abs(nu - c))
    l5 = np.maximum(np.abs(nr + c), np.abs(nu + c))
    l2, dp, dv = np.abs(nu), pr - pl, nr - nl
    c1, c2 = (l5 + l1) / 2 - l2, (l5 - l1) / 2
    k1, k2 = c1 * dp / c**2 + c2 * rho * dv / c, c1 * rho * dv + c2 * dp / c
    dis = [k1] + [k1 * u[a] + (k2 * sgn if a == r else 0) for a in range(d)] + [k1 * H + k2 * nu]
    return (fl + fr - sgn[:, None] * (l2[:, None] * (R - W) + np.stack(dis, axis=1))) / 2


def _exact_rhs(u, d, p, n, h, kind):
    """The residual [element, variable, node] on the periodic box of cells of size h."""
    n1 = p + 1
    gl, w = _gauss(n1)
    gll = _lobatto(n1)
    B, _ = _lagrange(gll, gl)
    Bi, D = _lagrange(gl, gll)[0], _lagrange(gl, gl)[1]      # D[j, i] = l_i'(x_j)
    Dw = (w[:, None] * D / w[None, :]).T
    end, _ = _lagrange(gl, np.array([-1, 1], dtype=L))
    u = u.astype(L).reshape((-1, d + 2) + (n1,) * d)
    s, out = u, 0
    for a in range(d):
        s = _along(B, s, a)
    for r in range(d):
        f, _, _ = _flux(s, d, r)
        y = _along(Dw, f, r)
        tr = []
        for side in (0, n1 - 1):   # traces: solution nodes on the face, interpolated along the other directions
            t = u
            for a in range(d):
                t = np.take(t, [side], axis=-1 - a) if a == r else _along(B, t, a)
            tr.append(t)
        cells = n[:d][::-1]
        right = np.roll(tr[0].reshape(cells + tr[0].shape[1:]), -1, axis=d - 1 - r).reshape(tr[0].shape)
        wrap = (np.arange(len(u)) // int(np.prod(n[:r])) % n[r] == n[r] - 1).reshape((-1, 1) + (1,) * d)
        F = _numflux(tr[1], right, d, r, kind, np.where(wrap, L(-1), L(1)))   # the + face of every element
        G = np.roll(F.reshape(cells + F.shape[1:]), 1, axis=d - 1 - r).reshape(F.shape)
        shape = [1] * y.ndim
        shape[-1 - r] = n1
        y = y - (end[1] / w).reshape(shape) * F + (end[0] / w).reshape(shape) * G
        out = out + y * 2 / L(h)
    for a in range(d):
        out = _along(Bi, out, a)
    return out.ravel()


CASES = {
    "quad-p1": (2, 1, (40, 40, 1), "Roe-Pike"), "quad-p2-lf": (2, 2, (24, 20, 1), "Lax-Friedrichs"),
    "quad-p3": (2, 3, (20, 16, 1), "Roe-Pike"), "quad-p4": (2, 4, (12, 12, 1), "Roe-Pike"),
    "hex-p1-lf": (3, 1, (8, 8, 6), "Lax-Friedrichs"), "hex-p2": (3, 2, (6, 5, 4), "Roe-Pike"),
    "hex-p2-lf": (3, 2, (6, 5, 4), "Lax-Friedrichs"), "hex-p3": (3, 3, (4, 4, 3), "Roe-Pike"),
}


@pytest.mark.parametrize("d,p,n,kind", list(CASES.values()), ids=list(CASES))
def test_rounding_of_the_residual(d, p, n, kind):
    torch = pytest.importorskip("torch")
    h = 0.25
    lo, hi = tuple(-h * k / 2 for k in n), tuple(h * k / 2 for k in n)
    cfg = dg.Config(d=d, p=p, n_elem=n, lo=lo, hi=hi, num_flux=kind, vortex=(4.0, 0.3, -0.2, 1.0, 0.8, 0.6, 0.0, 1.0))
    sim = dg.Simulation(cfg)
    u = sim.sol_coef()
    u = u * (1.0 + 1e-3 * np.random.default_rng(5).standard_normal(u.size))
    ctx = dg.GpuContext(sim)
    ctx.upload(u)
    ctx.compute_rhs()
    mesh, keep = _device_mesh(sim, cfg, torch)
    d_u = torch.from_numpy(u).cuda()
    d_r = torch.zeros_like(d_u)
    assert _entry()(C.byref(mesh), d_u.data_ptr(), d_r.data_ptr(), C.byref(C.c_double()), None) == 0
    ref = _exact_rhs(u, d, p, n, h, kind)
    assert u.size >= 5000 and np.max(np.abs(ctx.rhs() - ref)) <= 1e-11 * np.max(np.abs(ref))
    rms = [float(np.sqrt(np.mean((r - ref) ** 2))) for r in (ctx.rhs(), d_r.cpu().numpy())]
    print(f"rms error {rms[0]:.3e}, dense kernels {rms[1]:.3e}")
    assert rms[0] <= 1.1 * rms[1]
    del keep
