"""The two passes of an FP64 batch, problems for the tensor cores and for the FP64 loops."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("m,n", [(159, 64), (160, 63), (160, 64), (161, 65), (512, 63)])
def test_batched_line(tq, m, n):
    """Bar: least-squares solutions of N(0, 1) systems with 3 sqrt(m) on the diagonal (condition below 10),
    n reflectors: 32 sqrt(n) eps cond of the solution's norm."""
    import torch
    from tileqr import batched as Bt
    rng = np.random.default_rng(m + n)
    A0 = rng.standard_normal((m, n)) + 3 * np.sqrt(m) * np.eye(m, n)
    b = rng.standard_normal((m, 2))
    bg = Bt.BatchedGels(np.array([m], np.int32), np.array([n], np.int32), np.array([2], np.int32), dtype=torch.float64, tune=False)
    bg.load([A0], [b])
    bg.run()
    x = bg.x_view(0).cpu().numpy()
    ref = np.linalg.lstsq(A0, b, rcond=None)[0]
    assert np.linalg.norm(x - ref) <= 2 * 32 * np.sqrt(n) * EPS * 10 * np.linalg.norm(ref)


@pytest.mark.parametrize("replay", [False, True])
@pytest.mark.parametrize("nprob", [2, 40, 700])
def test_batched_passes_are_both_over_when_the_call_is(tq, nprob, replay):
    """Problems of the two passes, mixed: what follows on the stream sees all of them, and each has the bits it
    has in a batch of its own."""
    import torch
    from tileqr import batched as Bt
    sizes = [(512, 128, 3), (40, 20, 1), (160, 64, 2), (159, 100, 2), (300, 20, 1)]
    ms, ns, ks = (np.array([sizes[q % 5][j] for q in range(nprob)], np.int32) for j in range(3))
    g = torch.Generator(device="cuda").manual_seed(nprob)

    def solve(bg, A0, B0):
        out = []
        for _ in range(3):
            bg.A[:A0.numel()].copy_(A0)
            bg.B[:B0.numel()].copy_(B0)
            bg.replay(sync=False) if replay else bg.run(sync=False)
            out.append(bg.B.clone())
        assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
        return out[0]

    bg = Bt.BatchedGels(ms, ns, ks, dtype=torch.float64, tune=False)
    A0, B0 = (torch.randn(x.shape, generator=g, dtype=torch.float64, device="cuda") for x in (bg.A, bg.B))
    X = solve(bg, A0, B0)
    for q in range(min(nprob, 5)):
        one = Bt.BatchedGels(ms[q:q + 1], ns[q:q + 1], ks[q:q + 1], dtype=torch.float64, tune=False)
        a, b = int(bg.desc["a_off"][q]), int(bg.desc["b_off"][q])
        na, nb = int(ms[q]) * int(ns[q]), int(ms[q]) * int(ks[q])
        assert torch.equal(solve(one, A0[a:a + na], B0[b:b + nb])[:nb], X[b:b + nb])
