"""Strips of more than 256 rows that the tensor-core apply hands to the FP64 loops: the loops' staging of a
strip fits the shared memory the kernel has, and their results are the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def same(g, o):
    """Finite where the oracle is, and as close as sums of that many terms are in FP64 (suite bar for
    updates that grow)."""
    assert np.array_equal(np.isfinite(g), np.isfinite(o))
    f = np.isfinite(o)
    assert np.max(np.abs(g[f] - o[f]), initial=0.0) <= 1e-12 * np.max(np.abs(o[f]), initial=1.0)


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("m", [257, 300, 512])
@pytest.mark.parametrize("trans", ["C", "N"])
def test_tsmqr(tq, oracle, m, general, trans):
    rng = np.random.default_rng(m)
    k, ib, w = 64, 32, 40
    R, V = F(np.triu(rng.standard_normal((k, k)))), F(rng.standard_normal((m, k)))
    T, tau = np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.tsqrt(m, k, ib, R, V, T, tau, np.zeros(ib * k))
    A1, A2 = F(rng.standard_normal((k, w))), F(rng.standard_normal((m, w)))
    if general:                               # outside the bounds on V
        V, T = F(rng.uniform(-5, 5, (m, k))), F(np.triu(rng.uniform(-0.1, 0.1, (ib, k))))
    else:                                     # one column of one group, and all of a strip's
        A2[m - 1, 3] = np.nan
        A2[256, 16:32] = np.inf
    B1, B2 = tq.to_device(A1), tq.to_device(A2)
    tq.tsmqr("L", trans, k, w, m, w, k, ib, B1, B2, tq.to_device(V), tq.to_device(T), None)
    oracle.tsmqr("L", trans, k, w, m, w, k, ib, A1, A2, V, T, np.zeros(ib * w))
    same(np.vstack([tq.to_numpy(B1), tq.to_numpy(B2)]), np.vstack([A1, A2]))


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("m,k", [(257, 64), (300, 256), (512, 512)])
@pytest.mark.parametrize("trans", ["C", "N"])
def test_unmqr(tq, oracle, m, k, general, trans):
    rng = np.random.default_rng(m)
    ib, w = 32, 24
    V, T, tau = F(rng.standard_normal((m, k))), np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.geqrt(m, k, ib, V, T, tau, np.zeros(ib * k))
    C = F(rng.standard_normal((m, w)))
    if general:
        k = 64
        V, T = F(rng.uniform(-5, 5, (m, k))), F(np.triu(rng.uniform(-0.1, 0.1, (ib, k))))
    else:
        C[m - 1, 3] = np.nan
        C[5, 16:] = np.inf
    B = tq.to_device(C)
    tq.unmqr("L", trans, m, w, k, ib, tq.to_device(V), m, tq.to_device(T), B, None)
    oracle.unmqr("L", trans, m, w, k, ib, V, m, T, C, np.zeros((w, ib), order="F"))
    same(tq.to_numpy(B), C)
