"""FP64 Householder QR of matrices whose rows differ widely in size, heavy rows first: the light rows are
as accurate, each by its own size, as the heavy ones (the setting of weighted least squares and of equality
constraints by weighting), through every FP64 path that can use the tensor cores.

Bar: 16 times the error of plain FP64 loops (the oracle) on the same input, row by row against extended
precision, as heavy and light rows meet in a reflector's sums in an order that is each code's own, plus 32
sqrt(k) eps of the row's size for k reflectors (a rounding each, at random, and a factor of 32).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
WEIGHTS = [1.0, 1e3, 1e6, 1e12]


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def row_scales(m, weight, kind):
    """heavy: the first eight rows; graded: geometric from 1 down to 1 / weight."""
    s = np.ones(m)
    if kind == "heavy":
        s[:8] = weight
    else:
        s = weight ** (-np.arange(m) / max(1, m - 1))
    return s[:, None]


def apply_q(V, T, ib, C, trans, top=None):
    """Q^T C or Q C in extended precision; top None: V unit lower trapezoidal over C, else [I; V] over [top; C]."""
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


def row_error(x, y, size):
    """Largest error of a row, in units of that row's size."""
    e = np.max(np.abs((x - y).astype(np.float64)), axis=1)
    s = np.max(np.abs(np.asarray(size, dtype=np.float64)), axis=1)
    return float(np.max(e[s > 0] / s[s > 0])) if (s > 0).any() else 0.0


def bar(plain, k):
    return 16 * plain + 32 * np.sqrt(k) * EPS


@pytest.mark.parametrize("kind", ["heavy", "graded"])
@pytest.mark.parametrize("weight", WEIGHTS)
@pytest.mark.parametrize("m,k,ib,w", [(256, 32, 32, 16), (192, 96, 32, 24), (256, 256, 32, 8), (130, 64, 16, 9)])
def test_tsmqr_rows(tq, oracle, kind, weight, m, k, ib, w):
    """[R; A2] with R's rows (the first) heavy and A2's light, and columns scaled alike."""
    rng = np.random.default_rng(m + k)
    s = row_scales(k + m, weight, kind)
    R, V = F(np.triu(rng.standard_normal((k, k)) * s[:k])), F(rng.standard_normal((m, k)) * s[k:])
    T, tau = np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.tsqrt(m, k, ib, R, V, T, tau, np.zeros(ib * k))
    A1, A2 = F(rng.standard_normal((k, w)) * s[:k]), F(rng.standard_normal((m, w)) * s[k:])
    for trans in "CN":
        B1, B2 = tq.to_device(A1), tq.to_device(A2)
        tq.tsmqr("L", trans, k, w, m, w, k, ib, B1, B2, tq.to_device(V), tq.to_device(T), None)
        r2, r1 = apply_q(V, T, ib, A2, trans, A1)
        g, r, a = np.vstack([tq.to_numpy(B1), tq.to_numpy(B2)]), np.vstack([r1, r2]), np.vstack([A1, A2])
        size = np.hstack([a, r.astype(np.float64)])
        o1, o2 = A1.copy(order="F"), A2.copy(order="F")
        oracle.tsmqr("L", trans, k, w, m, w, k, ib, o1, o2, V, T, np.zeros(ib * w))
        assert row_error(g, r, size) <= bar(row_error(np.vstack([o1, o2]), r, size), k)


@pytest.mark.parametrize("kind", ["heavy", "graded"])
@pytest.mark.parametrize("weight", WEIGHTS)
@pytest.mark.parametrize("m,k,ib,w", [(256, 64, 32, 20), (256, 256, 32, 8), (400, 64, 32, 16), (160, 33, 16, 5)])
def test_unmqr_rows(tq, oracle, kind, weight, m, k, ib, w):
    """Q^T on columns scaled like the factored matrix; Q on the identity, whose zero rows become light ones."""
    rng = np.random.default_rng(2 * m + k)
    s = row_scales(m, weight, kind)
    V, T, tau = F(rng.standard_normal((m, k)) * s), np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.geqrt(m, k, ib, V, T, tau, np.zeros(ib * k))
    for trans, C in (("C", F(rng.standard_normal((m, w)) * s)), ("N", F(np.eye(m)[:, :w]))):
        B = tq.to_device(C)
        tq.unmqr("L", trans, m, w, k, ib, tq.to_device(V), m, tq.to_device(T), B, None)
        ref, _ = apply_q(V, T, ib, C, trans)
        size = np.hstack([C, ref.astype(np.float64)])
        o = C.copy(order="F")
        oracle.unmqr("L", trans, m, w, k, ib, V, m, T, o, np.zeros((w, ib), order="F"))
        assert row_error(tq.to_numpy(B), ref, size) <= bar(row_error(o, ref, size), k)


def check_factor(A0, A, T, nb, ib):
    """A0 = Q R row by row, Q from the flat tree's reflectors in extended precision."""
    m, n = A0.shape
    k = min(m, n)
    MT, KT = -(-m // nb), -(-k // nb)
    rows = [slice(i * nb, min(m, (i + 1) * nb)) for i in range(MT)]
    X = np.zeros((m, n), dtype=np.longdouble)
    X[:k] = np.triu(A[:k])
    for j in reversed(range(KT)):
        c = slice(j * nb, min(n, (j + 1) * nb))
        for i in reversed(range(j + 1, MT)):
            kk = min(rows[j].stop - rows[j].start, c.stop - c.start)
            X[rows[i]], X[rows[j]] = apply_q(A[rows[i], c][:, :kk], T[i * ib:, c][:, :kk], ib, X[rows[i]], "N", X[rows[j]])
        kk = min(rows[j].stop - rows[j].start, c.stop - c.start)
        X[rows[j]], _ = apply_q(A[rows[j], c][:, :kk], T[j * ib:, c][:, :kk], ib, X[rows[j]], "N")
    return row_error(X, A0, A0)


@pytest.mark.parametrize("dag", [True, False])
@pytest.mark.parametrize("kind", ["heavy", "graded"])
@pytest.mark.parametrize("weight", [1.0, 1e6, 1e12])
@pytest.mark.parametrize("m,n,nb,ib", [(256, 128, 128, 32), (512, 64, 256, 32), (300, 100, 256, 16)])
def test_tile_geqrf_rows(tq, oracle, dag, kind, weight, m, n, nb, ib):
    rng = np.random.default_rng(m + n)
    A0 = F(rng.standard_normal((m, n)) * row_scales(m, weight, kind))
    A = tq.to_device(A0)
    T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
    Ao = A0.copy(order="F")
    To, _ = oracle.tile_geqrf(Ao, nb, ib)
    assert check_factor(A0, tq.to_numpy(A), tq.to_numpy(T), nb, ib) <= bar(check_factor(A0, Ao, To, nb, ib), min(m, n))


@pytest.mark.parametrize("m,n,ib", [(256, 256, 32), (256, 32, 32), (200, 64, 16), (96, 96, 32)])
def test_triangular_tiles_keep_their_bits(tq, m, n, ib):
    """An upper triangular matrix has no reflectors: geqrt returns it as it is, entries far below their
    column's norm included."""
    rng = np.random.default_rng(n)
    A0 = F(np.triu(rng.standard_normal((m, n))))
    for j in range(0, n, 5):
        A0[j, j] = 1e-25 * (1 + j)
    graded = A0 * 2.0 ** -(np.arange(m) / 3.0)[:, None]
    for X in (A0, F(graded)):
        A, T, tau = tq.to_device(X), tq.zeros(ib, n), tq.zeros(n, 1)[:, 0]
        tq.geqrt(m, n, ib, A, T, tau, None)
        assert np.array_equal(tq.to_numpy(A), X)
        assert not tau.any()


@pytest.mark.parametrize("weight", WEIGHTS)
def test_weighted_least_squares(tq, oracle, weight):
    """Consistent weighted systems through the batched solver and the tile solver."""
    import torch
    from tileqr import batched as Bt
    m, n = 400, 64
    rng = np.random.default_rng(8)
    A0 = F(rng.standard_normal((m, n)) * row_scales(m, weight, "heavy"))
    x = rng.standard_normal((n, 2))
    b = F((A0.astype(np.longdouble) @ x.astype(np.longdouble)).astype(np.float64))
    plain = max(np.abs(oracle.tile_lstsq(A0[:h].copy(order="F"), b[:h].copy(order="F"), 256, 32) - x).max() for h in (m, 256))
    bg = Bt.BatchedGels(np.array([m, 256], np.int32), np.array([n, n], np.int32), np.array([2, 2], np.int32),
                        dtype=torch.float64, tune=False)
    bg.load([A0, A0[:256]], [b, b[:256]])
    bg.run()
    for q in range(2):
        assert np.abs(bg.x_view(q).cpu().numpy() - x).max() <= bar(plain, n)
    X = tq.tile_gels(tq.to_device(A0), tq.to_device(b), 256, 32)[0]
    assert np.abs(tq.to_numpy(X)[:n] - x).max() <= bar(plain, n)


@pytest.mark.parametrize("kind", ["heavy", "graded"])
@pytest.mark.parametrize("weight", WEIGHTS)
def test_differentiable_qr_rows(tq, oracle, kind, weight):
    import torch
    from tileqr import autodiff as AD
    m, n = 600, 96
    rng = np.random.default_rng(4)
    A0 = rng.standard_normal((2, m, n)) * row_scales(m, weight, kind)
    Q, R = AD.qr(torch.from_numpy(A0).cuda())
    for p in range(2):
        QR = Q[p].cpu().numpy().astype(np.longdouble) @ np.triu(R[p].cpu().numpy()).astype(np.longdouble)
        Qo, Ro, _ = oracle.qr_explicit(A0[p], 256, 32)
        plain = row_error(Qo.astype(np.longdouble) @ np.triu(Ro).astype(np.longdouble), A0[p], A0[p])
        assert row_error(QR, A0[p], A0[p]) <= bar(plain, n)


@pytest.mark.parametrize("weight", WEIGHTS)
@pytest.mark.parametrize("grp", [1, 4])
def test_tree_rows(tq, oracle, weight, grp):
    """The tree factorisation, through Q^T b and back-substitution."""
    m, n, nb, ib = 1024, 64, 128, 32
    rng = np.random.default_rng(6)
    A0 = F(rng.standard_normal((m, n)) * row_scales(m, weight, "heavy"))
    x = rng.standard_normal((n, 3))
    b = F((A0.astype(np.longdouble) @ x.astype(np.longdouble)).astype(np.float64))
    plain = np.abs(oracle.tile_lstsq(A0.copy(order="F"), b.copy(order="F"), nb, ib) - x).max()
    B = tq.to_device(b)
    A = tq.to_device(A0)
    T, tau, T2, tau2 = tq.tile_geqrf_tree(A, nb, ib, B=B, grp=grp)
    y = tq.to_numpy(B)[:n].astype(np.longdouble)
    R = np.triu(tq.to_numpy(A)[:n]).astype(np.longdouble)
    for r in range(n - 1, -1, -1):
        y[r] = (y[r] - R[r, r + 1:] @ y[r + 1:]) / R[r, r]
    assert np.abs(y.astype(np.float64) - x).max() <= bar(plain, n)
