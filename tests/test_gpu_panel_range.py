"""FP64 panels at scales where the square of a column's norm leaves the normal FP64 range, though no entry
does: the reflectors are then as right as the squares allow, or not finite; never wrong and finite.

The reference is the oracle on the same matrix scaled by a power of two into the middle of the range: V, T
and tau do not change, R scales.  Bar: the suite's 1e-12 max(m, n), plus what rounding squares of entries of
size s = 2^e to multiples of 2^-1074 does to their sum, 2^-1075 / s^2 a term relative to it, with a margin
of 64.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def ref_factor(oracle, A0, nb, ib):
    A = A0.copy(order="F")
    T, tau = oracle.tile_geqrf(A, nb, ib)
    return A, T, tau


@pytest.mark.parametrize("dag", [True, False])
@pytest.mark.parametrize("m,n,nb,ib", [(256, 32, 256, 32), (512, 64, 256, 32), (320, 48, 64, 16)])
@pytest.mark.parametrize("e", [-500, -508, -512, -515, -518, -522, -525, -528])
def test_subnormal_squares(tq, oracle, dag, m, n, nb, ib, e):
    rng = np.random.default_rng(m)
    A0 = F(rng.standard_normal((m, n)))
    Ao, To, tauo = ref_factor(oracle, A0, nb, ib)
    A = tq.to_device(np.ldexp(A0, e))
    T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
    bar = 1e-12 * max(m, n) + 64 * 2.0 ** (-1075 - 2 * e)
    A, T, tau = tq.to_numpy(A), tq.to_numpy(T), tq.to_numpy(tau)
    R = np.ldexp(np.triu(A[:n]), -e)
    V = A.copy()
    V[:n][np.triu_indices(n)] = 0
    Vo = Ao.copy()
    Vo[:n][np.triu_indices(n)] = 0
    assert np.abs(R - np.triu(Ao[:n])).max() <= bar * np.abs(Ao).max()
    assert np.abs(V - Vo).max() <= bar
    assert np.abs(T - To).max() <= bar * np.abs(To).max()
    assert np.abs(tau - tauo).max() <= 2 * bar


@pytest.mark.parametrize("dag", [True, False])
@pytest.mark.parametrize("e", [490, 500, 507, 511, 515, 600, 664])
def test_overflowing_squares(tq, oracle, dag, e):
    m, n, nb, ib = 512, 32, 256, 32
    rng = np.random.default_rng(e)
    A0 = F(rng.standard_normal((m, n)))
    Ao, To, tauo = ref_factor(oracle, A0, nb, ib)
    A = tq.to_device(np.ldexp(A0, e))
    T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
    A, tau = tq.to_numpy(A), tq.to_numpy(tau)
    if np.isfinite(A).all():
        assert np.abs(np.ldexp(np.triu(A[:n]), -e) - np.triu(Ao[:n])).max() <= 1e-12 * m * np.abs(Ao).max()
        assert np.abs(tau - tauo).max() <= 1e-12 * m
    else:
        assert e > 500                       # 2^500 sqrt(512) squares to 2^1009: in range
        assert not np.isfinite(A[0, :]).all()


@pytest.mark.parametrize("dag", [True, False])
def test_nearly_dependent_columns_of_a_small_matrix(tq, oracle, dag):
    """A column that is another one up to rounding, at 2^-470: what is left of it has subnormal squares.
    A = Q R column by column."""
    m, n, nb, ib = 512, 32, 256, 32
    rng = np.random.default_rng(1)
    A0 = F(rng.standard_normal((m, n)))
    A0[:, 12] = A0[:, 3] + np.ldexp(rng.standard_normal(m), -50)
    A0[:, 27] = A0[:, 20] * 3.0
    A0 = F(np.ldexp(A0, -470))
    A = tq.to_device(A0)
    T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
    X = tq.zeros(m, n)
    X[:n].copy_(A[:n].triu())
    tq.tile_unmqr("N", A, T, X, nb, ib)
    err = np.linalg.norm(np.ldexp(tq.to_numpy(X), 470) - np.ldexp(A0, 470), axis=0)
    assert (err <= 1e-14 * m * np.linalg.norm(np.ldexp(A0, 470), axis=0)).all()
    assert (tq.to_numpy(tau) <= 2.0 + 1e-10).all() and (tq.to_numpy(tau) >= 0).all()
