"""Which matrices that are not whole tiles are extended to whole ones, and what such a call leaves behind."""
import numpy as np
import pytest


def F(a):
    return np.array(a, dtype=np.float64, order="F")


@pytest.mark.parametrize("m,n,pays", [(65537, 1, False), (65537, 10, False), (4097, 33, False), (33, 4097, False),
                                      (257, 10, False), (520, 1, False), (200, 4097, False), (257, 257, False),
                                      (513, 513, True), (4000, 100, True), (65537, 129, True), (2900, 1500, True)])
def test_rule(m, n, pays):
    import tileqr
    assert tileqr._padded_pays(m, n, 256, 32) is pays


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(65537, 1), (20000, 10), (300, 40)])
def test_narrow_matrices_need_no_padded_copy(tq, m, n):
    import torch
    A = tq.to_device(F(np.random.default_rng(n).standard_normal((m, n))))
    (tr, tc), us = tq.tile_shapes(m, n, 256, 32)
    T, tau = tq.zeros(tr, tc), tq.zeros(*us)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    tq.tile_geqrf(A, 256, 32, T=T, tau=tau)
    assert torch.cuda.max_memory_allocated() - before < 8 * m * n


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,nb", [(65537, 1, 256), (300, 1, 128), (700, 129, 128), (129, 129, 128), (128, 129, 128), (513, 65, 64)])
def test_thin_and_barely_ragged_match_the_oracle(tq, oracle, m, n, nb):
    A0 = F(np.random.default_rng(m + n).standard_normal((m, n)))
    A = tq.to_device(A0)
    T, tau = tq.tile_geqrf(A, nb, 32)
    Ao = A0.copy(order="F")
    To, tauo = oracle.tile_geqrf(Ao, nb, 32)
    for x, y in ((A, Ao), (T, To), (tau, tauo)):
        assert np.max(np.abs(tq.to_numpy(x) - y)) <= 1e-12 * max(m, n) * np.max(np.abs(y))


@pytest.mark.gpu
def test_status_and_statistics_are_of_the_ragged_call(tq):
    """Also without blocking, where they are all that tells how the schedule ended."""
    import torch
    whole, ragged = (tq.to_device(F(np.random.default_rng(1).standard_normal(s))) for s in ((256, 128), (1000, 700)))
    tq.tile_geqrf(whole, 128, 32)
    tq.set_blocking(False)
    try:
        small = tq.dag_stats()
        tq.tile_geqrf(ragged, 128, 32)
        torch.zeros(64 << 20, device="cuda")            # whatever the call gave back is used again
        assert tq.dag_status()[0] == 0
        s = tq.dag_stats()
    finally:
        tq.set_blocking(True)
    assert s["busy_ms_TM"] > 0 and small["busy_ms_TM"] == 0


@pytest.mark.gpu
def test_matrices_that_require_gradients(tq):
    """The factorisation works on the memory of its arguments, in place, like the C entry points."""
    A0 = F(np.random.default_rng(2).standard_normal((300, 200)))
    out = []
    for grad in (False, True):
        A = tq.to_device(A0).requires_grad_(grad)
        T, tau = tq.tile_geqrf(A, 128, 32)
        out.append([tq.to_numpy(x) for x in (A, T, tau)])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
