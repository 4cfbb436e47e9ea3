"""An FP64 update of a column gives the same bits whatever columns share its strip and whichever driver runs
it, also for columns with a few entries far above the rest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def spiky(rng, m, n):
    """N(0, 1) columns, every third with one entry that makes up nearly all of its norm."""
    A = rng.standard_normal((m, n))
    for j in range(0, n, 3):
        A[rng.integers(m), j] = 100.0 * np.sqrt(m)
    return F(A)


@pytest.mark.parametrize("m,n,nb,ib", [(256, 256, 128, 32), (384, 256, 128, 8), (288, 192, 96, 24), (512, 256, 256, 16),
                                       (512, 512, 256, 8)])
@pytest.mark.parametrize("seed", range(3))
def test_drivers_agree_bit_for_bit(tq, m, n, nb, ib, seed):
    A0 = spiky(np.random.default_rng(seed), m, n)
    out = []
    for dag in (True, False):
        A = tq.to_device(A0)
        T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
        out.append([tq.to_numpy(x) for x in (A, T, tau)])
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("m,k,ib", [(256, 64, 32), (130, 40, 16), (300, 32, 32)])
def test_groups_of_eight_columns_stand_alone(tq, oracle, m, k, ib):
    """One call on 40 columns against calls on groups of eight of them."""
    rng = np.random.default_rng(m)
    R, V = F(np.triu(rng.standard_normal((k, k)))), F(rng.standard_normal((m, k)))
    T, tau = np.zeros((ib, k), order="F"), np.zeros(k)
    oracle.tsqrt(m, k, ib, R, V, T, tau, np.zeros(ib * k))
    A2 = spiky(rng, m, 40)
    A1 = F(rng.standard_normal((k, 40)))
    A2[:, 17] *= 1e-30                        # light rows beside heavy ones, and a column out of range
    A2[3, 30] = np.inf
    V, T = tq.to_device(V), tq.to_device(T)
    B1, B2 = tq.to_device(A1), tq.to_device(A2)
    tq.tsmqr("L", "C", k, 40, m, 40, k, ib, B1, B2, V, T, None)
    for c in range(0, 40, 8):
        C1, C2 = tq.to_device(A1[:, c:c + 8]), tq.to_device(A2[:, c:c + 8])
        tq.tsmqr("L", "C", k, 8, m, 8, k, ib, C1, C2, V, T, None)
        assert np.array_equal(tq.to_numpy(C1), tq.to_numpy(B1)[:, c:c + 8], equal_nan=True)
        assert np.array_equal(tq.to_numpy(C2), tq.to_numpy(B2)[:, c:c + 8], equal_nan=True)
