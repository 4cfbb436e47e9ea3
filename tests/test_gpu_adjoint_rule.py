"""Differentiable QR on either side of the line between the FP64 loops and the tensor cores."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("n,ib", [(31, 32), (32, 32), (32, 16), (40, 8), (127, 8), (128, 8), (12, 16)])
def test_differentiable_qr_line(tq, n, ib):
    """Bar: a rounding of the column's norm for each of n reflectors and each of the row tiles, at random,
    with a factor of 32."""
    import torch
    from tileqr import autodiff as AD
    A0 = np.random.default_rng(n).standard_normal((2, 300, n))
    Q, R = AD.qr(torch.from_numpy(A0).cuda(), ib)
    for p in range(2):
        q, r = Q[p].cpu().numpy().astype(np.longdouble), np.triu(R[p].cpu().numpy()).astype(np.longdouble)
        e = np.linalg.norm((q @ r - A0[p]).astype(np.float64), axis=0) / np.linalg.norm(A0[p], axis=0)
        assert e.max() <= 32 * np.sqrt(2 * n) * EPS
        o = np.linalg.norm((q.T @ q - np.eye(n)).astype(np.float64), axis=0)
        assert o.max() <= 32 * np.sqrt(2 * n) * EPS
