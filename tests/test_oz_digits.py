"""The digit products of the sliced FP64 residual (simplices) on the CPU: the lift operator of every supported element cut into
signed 8-bit digits as the library cuts it, and the largest magnitude each level's sum can reach with data digits at their
extremes (leading digit 64, the others 128).  An FP32 accumulator holds integers below 2^24 exactly.

Levels 0 to 4 are exact for every element; all levels for every element but the TET of order 4 (K = 439), whose levels 5, 6 and 7
stay below 1.5 x 2^24."""
import ctypes as C

import numpy as np
import pytest

import dpgsolver_gb300 as dg
from tests_support import DpgSim, _arr

S = 8
BIAS = sum(128 << (8 * i) for i in range(S - 1))


def _digits(a):
    """[S, rows, K] digits of the rows of a: a = sum_s d_s 2^(-8 s) 2^(E - 8), |a| 2^-E < 1/4."""
    E = np.frexp(np.abs(a).max(axis=1))[1] + 2
    n = np.rint(np.ldexp(a, 8 * S - E[:, None])).astype(np.int64) + BIAS   # below 2^63
    d = np.stack([n >> (8 * (S - 1))] + [((n >> (8 * (S - 1 - s))) & 255) - 128 for s in range(1, S)])
    return np.where(a == 0.0, 0, d)


def test_digits_restore_the_operator():
    a = np.random.default_rng(1).standard_normal((5, 40))
    d = _digits(a)
    E = np.frexp(np.abs(a).max(axis=1))[1] + 2
    back = sum(np.ldexp(d[s].astype(float), -8 * s) for s in range(S - 1, -1, -1))
    assert np.max(np.abs(np.ldexp(back, (E - 8)[:, None]) - a)) <= 2.0 ** -52 * np.max(np.abs(a))
    assert np.max(np.abs(d[0])) <= 64 and np.max(np.abs(d)) <= 128


CASES = [("tet", p, 0) for p in (1, 2, 3, 4)] + [("tet", 1, 4), ("tet", 2, 4), ("tri", 1, 4)] + [("tri", p, 0) for p in (2, 4, 5, 6, 7)]


@pytest.mark.parametrize("element,p,p_max", CASES, ids=[f"{e}-p{p}" + (f"to{q}" if q else "") for e, p, q in CASES])
def test_levels_are_exact(element, p, p_max):
    d = 3 if element == "tet" else 2
    sim = dg.Simulation(dg.Config(d=d, element=element, p=p, p_max=p_max, p_seed=3, n_elem=(4, 4, 4) if d == 3 else (8, 8, 1)))
    s = C.cast(sim.handle, C.POINTER(DpgSim)).contents
    nfc = {s.ops[k].p: s.ops[k].n_fc for k in range(s.n_ops)}
    most = np.array([64] + [128] * (S - 1))
    for k in range(s.n_ops):
        o = s.ops[k]
        n_s, n_c, n_fl = o.n_s, o.n_c, o.n_fl
        tw1 = _arr(o.tw1_vt_vc, d * n_s * n_c).reshape(d, n_s, n_c)
        parts, faces = [np.concatenate(list(tw1), axis=1)], []
        for pf in sorted(nfc):
            ptr = o.tw0_vt_fc if pf == o.p else o.tw0_vt_fcp[pf] if pf > o.p else None
            if ptr:
                t = _arr(ptr, n_fl * n_s * nfc[pf]).reshape(n_fl, n_s, nfc[pf])
                parts.append(-np.concatenate(list(t), axis=1))
                faces.append(nfc[pf])
        lift = _arr(o.m_inv_ref, n_s * n_s).reshape(n_s, n_s) @ np.concatenate(parts, axis=1)
        dig = np.abs(_digits(lift))
        level = np.stack([sum(dig[a] * most[L - a] for a in range(L + 1)) for L in range(S)], axis=-1)   # [row, K, level]
        total, off, face = level[:, :d * n_c].sum(axis=1), d * n_c, []
        for n in faces:   # a local face has one order: the largest of its parts
            face.append(np.stack([level[:, off + lf * n:off + (lf + 1) * n].sum(axis=1) for lf in range(n_fl)]))
            off += n_fl * n
        bound = (total + np.max(face, axis=0).sum(axis=0)).max(axis=0) / 2.0 ** 24
        assert np.all(bound[:5] < 1.0), bound
        assert np.all(bound < (1.5 if element == "tet" and o.p == 4 else 1.0)), bound
