"""The FP32 panels in registers (csrc/panel_reg.cuh) give the bits of the FP32 column step: the stream
driver's and the batched solver's factors at the edges of the register layout (8 columns a turn, 32 rows a
lane step, 256 and 512 rows) against the oracle, and against the same matrix factored with one more,
zero, column block, which moves the panel to another instantiation without changing any sum.
Bar: the suite's 1e-5 for FP32, times the square root of the column count (sums of that many roundings).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,nb,ib", [(20, 7, 32, 7), (33, 16, 33, 16), (63, 17, 63, 17), (130, 32, 50, 25),
                                       (300, 31, 256, 31), (512, 64, 256, 32), (200, 90, 100, 9)])
def test_fp32_panels_against_the_oracle(tq, oracle, m, n, nb, ib):
    import torch
    rng = np.random.default_rng(m * n)
    A0 = np.array(rng.standard_normal((m, n)), dtype=np.float32, order="F")
    A = tq.to_device(A0, dtype=torch.float32)
    T, tau = tq.tile_geqrf(A, nb, ib, dag=False)
    Ao = np.array(A0, dtype=np.float64, order="F")
    To, tauo = oracle.tile_geqrf(Ao, nb, ib)
    for x, y in ((A, Ao), (T, To), (tau, tauo)):
        x = tq.to_numpy(x).astype(np.float64)
        assert np.linalg.norm(x - y) <= 1e-5 * np.sqrt(n) * np.linalg.norm(y)


@pytest.mark.parametrize("m,n", [(40, 9), (256, 16), (200, 13)])
def test_instantiations_agree_bit_for_bit(tq, m, n):
    """ib = n <= 16 columns a panel (two columns a warp) against ib = n + 16 with 16 zero columns appended
    (four columns a warp, the same sums)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    A0 = tq.empty(m, n, dtype=torch.float32)
    A0.copy_(torch.randn(m, n, generator=g, device="cuda"))
    A = A0.clone()
    T, tau = tq.tile_geqrf(A, 256, n, dag=False)
    B = tq.zeros(m, n + 16, dtype=torch.float32)
    B[:, :n].copy_(A0)
    T2, tau2 = tq.tile_geqrf(B, 256, n + 16, dag=False)
    assert torch.equal(A, B[:, :n])
    assert torch.equal(tau[:n], tau2[:n])
    assert torch.equal(torch.triu(T[:n, :n]), torch.triu(T2[:n, :n]))


@pytest.mark.parametrize("m", [255, 257, 300, 511, 512])
def test_batched_rows_beyond_one_chunk(tq, m):
    """Panels of more than 256 rows: two row chunks a lane, through the batched solver."""
    import torch
    from tileqr import batched as Bt
    ms, ns, ks = np.array([m, m], np.int32), np.array([min(m, 40), 16], np.int32), np.array([2, 1], np.int32)
    bg = Bt.BatchedGels(ms, ns, ks, dtype=torch.float32)
    rng = np.random.default_rng(m)
    As = [rng.standard_normal((m, n)) for n in ns]
    Bs = [rng.standard_normal((m, k)) for k in ks]
    bg.load(As, Bs)
    bg.run()
    for q in range(2):
        x = bg.x_view(q).double().cpu().numpy()
        ref = np.linalg.lstsq(np.float32(As[q]).astype(np.float64), np.float32(Bs[q]).astype(np.float64), rcond=None)[0]
        assert np.linalg.norm(x - ref) <= 1e-5 * np.sqrt(ns[q]) * np.linalg.norm(ref)
