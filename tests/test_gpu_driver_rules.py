"""Where the FP64 tile drivers change between two CTAs per SM on the FP64 loops and one on the tensor cores:
on either side of the line the task graph and the stream driver give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def F(a):
    return np.array(a, dtype=np.float64, order="F")


@pytest.mark.parametrize("n_tiles", [1, 3])
@pytest.mark.parametrize("nb,ib", [(64, 16), (64, 32), (72, 24), (80, 16), (96, 16), (112, 16), (128, 16), (256, 8), (192, 8)])
def test_task_graph_and_stream_driver_agree(tq, nb, ib, n_tiles):
    A0 = F(np.random.default_rng(nb + ib).standard_normal((3 * nb, n_tiles * nb)))
    out = []
    for dag in (True, False):
        A = tq.to_device(A0)
        T, tau = tq.tile_geqrf(A, nb, ib, dag=dag)
        out.append([tq.to_numpy(x) for x in (A, T, tau)])
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("rhs", [0, 3])
@pytest.mark.parametrize("m,n,nb,ib", [(256, 64, 64, 16), (256, 128, 64, 16), (300, 96, 96, 16), (512, 200, 200, 10),
                                       (700, 256, 256, 8), (700, 300, 256, 8), (512, 128, 128, 16)])
def test_tree_drivers_agree(tq, m, n, nb, ib, rhs):
    rng = np.random.default_rng(m + n)
    A0, B0 = F(rng.standard_normal((m, n))), F(rng.standard_normal((m, max(rhs, 1))))
    out = []
    for dag in (True, False):
        A, B = tq.to_device(A0), tq.to_device(B0) if rhs else None
        T = tq.tile_geqrf_tree(A, nb, ib, B=B, dag=dag)
        out.append([tq.to_numpy(x) for x in (A, *T, *([B] if rhs else []))])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
