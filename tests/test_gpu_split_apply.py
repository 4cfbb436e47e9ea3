"""The FP64 block-reflector apply on the tensor cores (csrc/oz_apply.cuh), against extended precision.

The sizes are the edges of its warps, digit blocks and strips.  Reflectors come from the oracle's
factorisations, so the updates are orthogonal and the expected error of a column is a few roundings of
its norm: the bar is 32 sqrt(k) eps of the column's norm (k reflectors, each moving an element by one
rounding of the column's size, with a margin of 32), on both sides of the comparison's own 64-bit
reference being extended precision.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def reflectors_ge(oracle, m, k, ib, rng):
    A, T, tau = F(rng.standard_normal((m, k))), np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.geqrt(m, k, ib, A, T, tau, np.zeros(ib * k))
    return A, T


def reflectors_ts(oracle, m, k, ib, rng):
    R, V = F(np.triu(rng.standard_normal((k, k)))), F(rng.standard_normal((m, k)))
    T, tau = np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.tsqrt(m, k, ib, R, V, T, tau, np.zeros(ib * k))
    return V, T


def reflectors_tt(oracle, k, ib, rng):
    R, V = F(np.triu(rng.standard_normal((k, k)))), F(np.triu(rng.standard_normal((k, k))))
    T, tau = np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.ttqrt(k, k, ib, R, V, T, tau, np.zeros(ib * k))
    return V, T


def apply_ref(V, T, ib, C, trans, top):
    """Q^T C or Q C in extended precision; V m x k with its leading part implicit in `top` form:
    top None: V itself unit lower trapezoidal over C; else [I; V] over [top; C]."""
    L = np.longdouble
    C, k = C.astype(L), V.shape[1]
    top = None if top is None else top.astype(L)
    blocks = list(range(0, k, ib))
    for i in (blocks if trans == "C" else blocks[::-1]):
        kb = min(ib, k - i)
        Tb = np.triu(T[:kb, i:i + kb]).astype(L)
        Tb = Tb.T if trans == "C" else Tb
        if top is None:
            Vb = np.tril(V[:, i:i + kb].astype(L), -1 - i)
            Vb[np.arange(i, i + kb), np.arange(kb)] = 1
            C -= Vb @ (Tb @ (Vb.T @ C))
        else:
            Vb = V[:, i:i + kb].astype(L)
            W = Tb @ (top[i:i + kb] + Vb.T @ C)
            top[i:i + kb] -= W
            C -= Vb @ W
    return C, top


def worst(x, y, norms):
    return float(np.max(np.linalg.norm((x - y).astype(np.float64), axis=0) / norms))


@pytest.mark.parametrize("m,k,ib,w", [(64, 33, 32, 1), (128, 32, 32, 16), (129, 64, 16, 17), (100, 70, 24, 5),
                                      (255, 256, 32, 31), (256, 256, 32, 48), (121, 35, 17, 16),
                                      (256, 16, 16, 40), (127, 32, 32, 3), (257, 64, 32, 17),
                                      (300, 40, 16, 16), (512, 256, 32, 33)])
def test_tsmqr_every_edge(tq, oracle, m, k, ib, w):
    rng = np.random.default_rng(m + k)
    V, T = reflectors_ts(oracle, m, k, ib, rng)
    A1, A2 = F(rng.standard_normal((k, w))), F(rng.standard_normal((m, w)))
    norms = np.sqrt((A1 ** 2).sum(0) + (A2 ** 2).sum(0))
    for side in "LR":
        for trans in "CN":
            B1, B2 = (tq.to_device(A1 if side == "L" else A1.T), tq.to_device(A2 if side == "L" else A2.T))
            # C op(Q) is (op(Q)^T C^T)^T
            tq.tsmqr(side, trans, *B1.shape, *B2.shape, k, ib, B1, B2, tq.to_device(V), tq.to_device(T), None)
            lt = trans if side == "L" else ("N" if trans == "C" else "C")
            r2, r1 = apply_ref(V, T, ib, A2, lt, A1)
            g1, g2 = tq.to_numpy(B1), tq.to_numpy(B2)
            if side == "R":
                g1, g2 = g1.T, g2.T
            bar = 32 * np.sqrt(k) * EPS
            assert worst(np.vstack([g1, g2]), np.vstack([r1, r2]), norms) <= bar


@pytest.mark.parametrize("m,k,ib,w", [(128, 32, 32, 3), (130, 40, 16, 16), (256, 200, 32, 33), (200, 199, 31, 16),
                                      (256, 256, 8, 16), (290, 280, 32, 20), (512, 512, 32, 16), (511, 31, 31, 33)])
def test_unmqr_every_edge(tq, oracle, m, k, ib, w):
    rng = np.random.default_rng(3 * m + k)
    V, T = reflectors_ge(oracle, m, k, ib, rng)
    C = F(rng.standard_normal((m, w)))
    for trans in "CN":
        B = tq.to_device(C)
        tq.unmqr("L", trans, m, w, k, ib, tq.to_device(V), m, tq.to_device(T), B, None)
        ref, _ = apply_ref(V, T, ib, C, trans, None)
        assert worst(tq.to_numpy(B), ref, np.linalg.norm(C, axis=0)) <= 32 * np.sqrt(k) * EPS


def test_ttmqr_leaves_rows_past_the_triangle(tq, oracle):
    """Rows below the last reflector's triangle are another factor's: they keep their bits, whatever
    they hold, and do not enter the column scales."""
    rng = np.random.default_rng(4)
    k, ib, m, w = 40, 16, 128, 20
    V, T = reflectors_tt(oracle, k, ib, rng)
    Vm = np.zeros((m, k), order="F")
    Vm[:k] = np.triu(V) + np.tril(rng.standard_normal((k, k)) * 1e300, -1)
    A1, A2 = F(rng.standard_normal((k, w))), F(rng.standard_normal((m, w)))
    A2[k:] = np.where(rng.random((m - k, w)) < 0.5, np.inf, 1e-310)
    B1, B2 = tq.to_device(A1), tq.to_device(A2)
    tq.ttmqr("L", "C", k, w, m, w, k, ib, B1, B2, tq.to_device(Vm), tq.to_device(T), None)
    ref2, ref1 = apply_ref(np.triu(V), T, ib, A2[:k], "C", A1)
    g1, g2 = tq.to_numpy(B1), tq.to_numpy(B2)
    norms = np.sqrt((A1 ** 2).sum(0) + (A2[:k] ** 2).sum(0))
    assert worst(np.vstack([g1, g2[:k]]), np.vstack([ref1, ref2]), norms) <= 32 * np.sqrt(k) * EPS
    assert np.array_equal(g2[k:], A2[k:])


@pytest.mark.parametrize("scale", [1e-300, 1e-200, 1.0, 1e200, 1e306])
def test_scales_zeros_and_nonfinite_columns(tq, oracle, scale):
    """Columns far apart in size, zero, sparse, subnormal and non-finite ones in one strip: each column
    as accurate as alone, a column no reflector meets unchanged, and the strips outside the fixed-point
    range agree with the oracle on which entries are finite."""
    rng = np.random.default_rng(11)
    m, k, ib, w = 96, 64, 32, 64
    V, T = reflectors_ts(oracle, m, k, ib, rng)
    A1, A2 = F(rng.standard_normal((k, w))), F(rng.standard_normal((m, w)))
    A1 *= scale
    A2 *= scale
    for j in (1, 17, 33):
        A1[:, j], A2[:, j] = A1[:, j] * 2.0 ** -60, A2[:, j] * 2.0 ** -60
    A1[:, 2] = A2[:, 2] = 0.0
    A1[:, 3], A2[:, 3] = 0.0, 0.0
    A2[7, 3] = scale
    A2[5, 20] = np.nan                        # strip 1: a NaN
    A1[9, 40] = np.inf                        # strip 2: an infinity
    A1[:, 50], A2[:, 50] = 5e-320, 5e-320     # strip 3: subnormals
    B1, B2 = tq.to_device(A1), tq.to_device(A2)
    tq.tsmqr("L", "C", k, w, m, w, k, ib, B1, B2, tq.to_device(V), tq.to_device(T), None)
    g = np.vstack([tq.to_numpy(B1), tq.to_numpy(B2)])
    o1, o2 = A1.copy(order="F"), A2.copy(order="F")
    oracle.tsmqr("L", "C", k, w, m, w, k, ib, o1, o2, V, T, np.zeros(ib * w))
    o = np.vstack([o1, o2])
    assert np.array_equal(np.isfinite(g), np.isfinite(o))
    assert np.all(g[:, 2] == 0.0)
    cols = [j for j in range(w) if j not in (2, 20, 40, 50)]
    with np.errstate(all="ignore"):
        r2, r1 = apply_ref(V, T, ib, A2[:, cols], "C", A1[:, cols])
        norms = np.sqrt((A1[:, cols].astype(np.longdouble) ** 2).sum(0) + (A2[:, cols].astype(np.longdouble) ** 2).sum(0))
        d = np.sqrt(((g[:, cols] - np.vstack([r1, r2])) ** 2).sum(0))
    # plus one unit of the subnormal range per rounding: it is all a column of such numbers resolves
    assert np.all(d <= 32 * np.sqrt(k) * EPS * norms + k * np.sqrt(m + k) * np.longdouble(2) ** -1074)


def test_general_v_and_t_match_the_oracle(tq, oracle):
    """V and T that are no reflectors: outside the bounds, or inside them with a growing result."""
    rng = np.random.default_rng(12)
    m, k, ib, w = 128, 64, 32, 20
    for vs, ts in ((5.0, 0.1), (1.0, 3.9), (1.9, 1.0), (0.05, 100.0), (np.inf, 1.0)):
        V = F(rng.uniform(-1, 1, (m, k)) * (1.0 if np.isinf(vs) else vs))
        if np.isinf(vs):
            V[3, 4] = np.nan
        T = F(np.triu(rng.uniform(-1, 1, (ib, k))) * ts)
        A1, A2 = F(rng.standard_normal((k, w))), F(rng.standard_normal((m, w)))
        B1, B2 = tq.to_device(A1), tq.to_device(A2)
        tq.tsmqr("L", "C", k, w, m, w, k, ib, B1, B2, tq.to_device(V), tq.to_device(T), None)
        oracle.tsmqr("L", "C", k, w, m, w, k, ib, A1, A2, V, T, np.zeros(ib * w))
        g, o = np.vstack([tq.to_numpy(B1), tq.to_numpy(B2)]), np.vstack([A1, A2])
        assert np.array_equal(np.isfinite(g), np.isfinite(o))
        f = np.isfinite(o)
        # the growth of two blocks of general W = T (A1 + V^T A2): compare with the largest result
        assert np.max(np.abs(g[f] - o[f]), initial=0.0) <= 1e-12 * np.max(np.abs(o[f]), initial=1.0)
