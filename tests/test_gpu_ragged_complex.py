"""Complex matrices that are not whole tiles, through the default entry (dag=True): the oracle's factor, the
reference's rule for a column of one row (no reflector) included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["complex128", "complex64"])
@pytest.mark.parametrize("m,n,nb,ib", [(300, 300, 128, 32), (300, 500, 128, 32), (257, 700, 128, 32), (257, 257, 256, 32),
                                       (300, 200, 128, 32), (256, 300, 128, 32), (100, 130, 64, 16)])
def test_ragged_complex_matches_the_oracle(tq, oracle, dt, m, n, nb, ib):
    import torch
    rng = np.random.default_rng(m + n)
    A0 = np.asfortranarray((rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))).astype(dt).astype(np.complex128))
    A = tq.to_device(A0, dtype=getattr(torch, dt))
    T, tau = tq.tile_geqrf(A, nb, ib)
    Ao = A0.copy(order="F")
    To, tauo = oracle.tile_geqrf(Ao, nb, ib)
    bar = (1e-12 if dt == "complex128" else 1e-4) * max(m, n)
    for x, y in ((A, Ao), (T, To), (tau, tauo)):
        x = tq.to_numpy(x).astype(np.complex128)
        assert np.abs(x - y).max() <= bar * np.abs(y).max()
    assert np.array_equal(tq.to_numpy(tau) == 0, tauo == 0)
