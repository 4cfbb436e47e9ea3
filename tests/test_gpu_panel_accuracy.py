"""The FP64 panels (csrc/panel_blk.cuh) column by column against extended precision, and the FP32 ones
(csrc/panel_reg.cuh) bit for bit against the column step that wider panels take.

Bars: k reflectors, each a rounding of the column's norm at random, and a factor of 32.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
L = np.longdouble


def F(a):
    return np.array(a, dtype=np.float64, order="F")


def check(A0, V, R, T, tau, k):
    """A0 = (I - V T V^T) [R; 0], tau = 2 / |v|^2 and T larft's, from the computed V in extended precision."""
    bar = 32 * np.sqrt(k) * EPS
    V, T, n = V.astype(L), np.triu(T).astype(L), A0.shape[1]
    X = np.zeros(A0.shape, dtype=L)
    X[:R.shape[0]] = R
    X -= V @ (T @ (V.T @ X))
    assert np.max(np.linalg.norm((X - A0).astype(np.float64), axis=0) / np.linalg.norm(A0, axis=0)) <= bar
    G = V.T @ V
    t = 2 / np.diagonal(G)
    assert np.max(np.abs(tau - t)) <= bar
    # T^-1 + T^-T = V^T V, multiplied out
    D = T + T.T - T.T @ G @ T
    assert np.max(np.abs(D.astype(np.float64))) <= 4 * bar


@pytest.mark.parametrize("m,nc", [(64, 9), (65, 16), (127, 17), (129, 24), (200, 25), (255, 32), (256, 32), (256, 10),
                                  (257, 32), (400, 31), (512, 32)])
def test_geqrt_and_tsqrt(tq, m, nc):
    rng = np.random.default_rng(m + nc)
    A0, R0 = F(rng.standard_normal((m, nc))), F(np.triu(rng.standard_normal((nc, nc))))
    A, T, tau = tq.to_device(A0), tq.zeros(nc, nc), tq.zeros(nc, 1)[:, 0]
    tq.geqrt(m, nc, nc, A, T, tau, None)
    A = tq.to_numpy(A)
    V = np.tril(A, -1)
    V[np.arange(nc), np.arange(nc)] = 1
    check(A0, V, np.triu(A[:nc]), tq.to_numpy(T), tau.cpu().numpy(), nc)
    A, R, T, tau = tq.to_device(A0), tq.to_device(R0), tq.zeros(nc, nc), tq.zeros(nc, 1)[:, 0]
    tq.tsqrt(m, nc, nc, R, A, T, tau, None)
    V = np.vstack([np.eye(nc), tq.to_numpy(A)])
    check(np.vstack([R0, A0]), V, np.triu(tq.to_numpy(R)), tq.to_numpy(T), tau.cpu().numpy(), nc)


@pytest.mark.parametrize("m,n", [(20, 7), (63, 17), (256, 32), (512, 32), (300, 31), (400, 16), (200, 9), (257, 24)])
def test_fp32_panels_have_the_bits_of_the_column_step(tq, m, n):
    """n <= 32 columns a panel against the same columns followed by zero ones, 40 in all, which no sum meets."""
    import torch
    A0 = np.random.default_rng(m * n).standard_normal((m, n)).astype(np.float32)
    A = tq.to_device(np.asfortranarray(A0), dtype=torch.float32)
    T, tau = tq.tile_geqrf(A, 256, n, dag=False)
    B = tq.zeros(m, 40, dtype=torch.float32)
    B[:, :n].copy_(torch.from_numpy(A0).cuda())
    T2, tau2 = tq.tile_geqrf(B, 256, 40, dag=False)
    assert torch.equal(A, B[:, :n])
    assert torch.equal(tau[:n], tau2[:n])
    k = min(m, n)
    for i in range(-(-m // 256)):
        a, b = T[i * n:i * n + k, :k], T2[i * 40:i * 40 + k, :k]
        assert torch.equal(torch.triu(a), torch.triu(b))
