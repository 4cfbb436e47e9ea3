"""The blocked FP64 column loop of the panels (csrc/panel_blk.cuh) against the oracle, at the edges of its
sub-blocks of eight columns, its warps of 32 rows and its 256-row chunks; and matrices that are not whole
tiles through the persistent kernel.  Bars: the suite's 1e-12 max(m, n), relative to the largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def close(a, b, tol, scale=None):
    s = np.max(np.abs(b)) if scale is None else scale
    return np.max(np.abs(a - b)) <= tol * max(s, 1e-300)


def factor(tq, A0, nb, ib, dag):
    A = tq.to_device(A0)
    T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
    return [tq.to_numpy(x) for x in (A, T, tau)]


@pytest.mark.parametrize("dag", [False, True])
@pytest.mark.parametrize("m,n,nb,ib", [(64, 9, 64, 9), (129, 17, 65, 17), (200, 24, 128, 24), (321, 32, 256, 32),
                                       (255, 31, 255, 31), (512, 40, 256, 32), (777, 50, 256, 16), (300, 130, 96, 12)])
def test_panel_edges(tq, oracle, dag, m, n, nb, ib):
    rng = np.random.default_rng(m + n)
    A0 = F(rng.standard_normal((m, n)))
    Ao = A0.copy(order="F")
    To, tauo = oracle.tile_geqrf(Ao, nb, ib)
    for x, y in zip(factor(tq, A0, nb, ib, dag), (Ao, To, tauo)):
        assert close(x, y, 1e-12 * max(m, n))


@pytest.mark.parametrize("m,n", [(1000, 500), (257, 700), (513, 256), (700, 300), (255, 513)])
def test_ragged_matrices_on_the_persistent_kernel(tq, oracle, m, n):
    """Extended to whole tiles inside: the same factor as the oracle's, and what the call does not write
    (T and tau of columns without a tile above the diagonal, padding of a wider T) is left as it was."""
    nb, ib = 128, 32
    rng = np.random.default_rng(m)
    A0 = F(rng.standard_normal((m, n)))
    (tr, tc), (ur, uc) = tq.tile_shapes(m, n, nb, ib)
    T0, tau0 = F(rng.standard_normal((tr + 3, tc + 2))), F(rng.standard_normal((ur, uc)))
    out = []
    for dag in (True, False):
        A, T, tau = tq.to_device(A0), tq.to_device(T0), tq.to_device(tau0)
        tq.tile_geqrf(A, nb, ib, T=T, tau=tau, dag=dag)
        out.append([tq.to_numpy(x) for x in (A, T, tau)])
    Ao = A0.copy(order="F")
    oracle.tile_geqrf(Ao, nb, ib)
    assert close(out[0][0], Ao, 1e-12 * max(m, n))
    for x, y, x0 in zip(out[0], out[1], (A0, T0, tau0)):
        assert close(x, y, 1e-12 * max(m, n))
        assert np.array_equal(x == x0, y == x0)


def test_zero_repeated_and_scaled_columns(tq, oracle):
    """Zero columns (no reflector, T's column left), columns that become zero, and scales the fixed point
    holds or hands back to the FP64 loop."""
    rng = np.random.default_rng(3)
    m, n, nb, ib = 512, 32, 256, 32
    for scale in (1.0, 1e-120, 1e150, 1e-300):
        A0 = F(rng.standard_normal((m, n))) * scale
        A0[:, 3] = 0.0
        A0[:, 11] = 0.0
        A0[256:, 20] = 0.0
        A0[:, 25] *= 1e-9
        Ao = A0.copy(order="F")
        To, tauo = oracle.tile_geqrf(Ao, nb, ib)
        for dag in (True, False):
            A, T, tau = factor(tq, A0, nb, ib, dag)
            assert np.array_equal(tau == 0, tauo == 0)
            norms = np.linalg.norm(Ao / scale, axis=0) * scale
            big = norms > 0
            assert np.max(np.abs(np.triu(A[:n]) - np.triu(Ao[:n]))[:, big] / norms[big]) <= 1e-12 * m
            assert close(T, To, 1e-12 * m) and close(tau, tauo, 1e-12 * m)


def test_nonfinite_panel(tq, oracle):
    rng = np.random.default_rng(5)
    A0 = F(rng.standard_normal((512, 32)))
    A0[300, 12] = np.nan
    Ao = A0.copy(order="F")
    oracle.tile_geqrf(Ao, 256, 32)
    for dag in (True, False):
        A, T, tau = factor(tq, A0, 256, 32, dag)
        assert np.array_equal(np.isfinite(A), np.isfinite(Ao))
