"""The workloads the library's speed is judged by, each one pass through its public entry points.

A case is a dict of plain values; `listed()` gives the standing ones, `draw(rng)` another of the same
ranges.  `prepare` makes what a program has in hand (device matrices, a batch plan), `run` is one pass,
`work` the bytes and flops a pass cannot do without, `exact` the same results in 64 bits from plain
torch, where that takes seconds.

The tile factorisations work in place, so a pass first copies the input into the working matrix, as a
program that keeps its A does.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nextla.jl_gb300"))

import tileqr as tq  # noqa: E402
from tileqr import autodiff, batched  # noqa: E402

DTYPES = {"f64": torch.float64, "f32": torch.float32, "c128": torch.complex128}


def listed():
    return [
        # the drop-in use of the tile kernels: one tile step (geqrt, unmqr, tsqrt, tsmqr) called routine by
        # routine, as an external scheduler does; small FP32 tiles are the smallest calls
        {"name": "tile_step_f32_64", "kind": "tile", "dtype": "f32", "nb": 64, "ib": 16, "w": 64, "m2": 64},
        {"name": "tile_step_f64_256", "kind": "tile", "dtype": "f64", "nb": 256, "ib": 32, "w": 256, "m2": 256},
        # a mid-size solve step: QR of one 1024 x 1024 matrix and Q^T on 16 right-hand sides
        {"name": "qr_f64_1024_rhs16", "kind": "qr", "dtype": "f64", "m": 1024, "n": 1024, "nb": 256, "ib": 32, "rhs": 16},
        # a ragged matrix: no dimension is a multiple of the tile
        {"name": "qr_f64_2900x1500", "kind": "qr", "dtype": "f64", "m": 2900, "n": 1500, "nb": 256, "ib": 32, "rhs": 0},
        # the large square factorisation, double and single precision, and a complex one
        {"name": "qr_f64_8192", "kind": "qr", "dtype": "f64", "m": 8192, "n": 8192, "nb": 256, "ib": 32, "rhs": 0},
        {"name": "qr_f32_4096", "kind": "qr", "dtype": "f32", "m": 4096, "n": 4096, "nb": 256, "ib": 32, "rhs": 0},
        {"name": "qr_c128_2048", "kind": "qr", "dtype": "c128", "m": 2048, "n": 2048, "nb": 256, "ib": 32, "rhs": 0},
        # tall and skinny, through the hierarchical reduction tree
        {"name": "tall_f64_65536x512", "kind": "tall", "dtype": "f64", "m": 65536, "n": 512, "nb": 256, "ib": 32, "grp": 4},
        # least squares: mixed precision (FP32 matrix, FP64 solution) on an ill-conditioned matrix
        {"name": "lstsq_mixed_32768x4096", "kind": "mixed", "m": 32768, "n": 4096, "k": 4, "nb": 256, "ib": 32},
        # a batch of small uneven least-squares problems, double and single precision
        {"name": "batched_f64_4096", "kind": "batched", "dtype": "f64", "nprob": 4096, "max_m": 512},
        {"name": "batched_f32_4096", "kind": "batched", "dtype": "f32", "nprob": 4096, "max_m": 512},
        # differentiable QR: thin Q and R of a batch, and the gradient for given cotangents
        {"name": "diffqr_f64_256x2048x256", "kind": "diffqr", "dtype": "f64", "batch": 256, "m": 2048, "n": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tile", "qr", "qr", "tall", "mixed", "batched", "diffqr"])
    if kind == "tile":
        nb = _log(rng, 32, 256)
        return {"kind": kind, "dtype": rng.choice(["f64", "f64", "f32", "c128"]), "nb": nb,
                "ib": rng.choice([8, 16, 24, 32]), "w": _log(rng, 1, 512), "m2": rng.randint(nb // 2, nb)}
    if kind == "qr":
        dtype = rng.choice(["f64", "f64", "f32", "c128"])
        top = {"f64": 8192, "f32": 8192, "c128": 2048}[dtype]
        m, n = _log(rng, 256, top), _log(rng, 256, top)
        if rng.random() < 0.5:                       # whole tiles
            m, n = max(256, m // 256 * 256), max(256, n // 256 * 256)
        return {"kind": kind, "dtype": dtype, "m": m, "n": n, "nb": 256, "ib": rng.choice([16, 32, 32]),
                "rhs": rng.choice([0, 1, 4, 16])}
    if kind == "tall":
        return {"kind": kind, "dtype": "f64", "m": _log(rng, 2048, 65536), "n": _log(rng, 64, 512), "nb": 256,
                "ib": 32, "grp": rng.choice([1, 2, 4, 8])}
    if kind == "mixed":
        n = 256 * rng.randint(1, 12)
        return {"kind": kind, "m": n * rng.randint(2, 8), "n": n, "k": rng.randint(1, 8), "nb": 256, "ib": 32}
    if kind == "batched":
        return {"kind": kind, "dtype": rng.choice(["f64", "f32"]), "nprob": _log(rng, 128, 4096),
                "max_m": _log(rng, 48, 512)}
    n = rng.randint(16, 256)
    return {"kind": kind, "dtype": "f64", "batch": _log(rng, 16, 256), "m": rng.randint(max(n + 1, 256), 2048), "n": n}


# ---- inputs -----------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(shape, dtype, g):
    if dtype.is_complex:
        return torch.complex(torch.randn(shape, generator=g, dtype=torch.float64, device="cuda"),
                             torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")).to(dtype)
    return torch.randn(shape, generator=g, dtype=torch.float64, device="cuda").to(dtype)


def _matrix(m, n, dtype, g):
    """Column-major m x n matrix of N(0, 1) entries."""
    return _randn((n, m), dtype, g).t()


def _mix_rows(X, g, rounds=4, blk=64):
    """Multiplies X from the left by a random orthogonal matrix: rounds of a row permutation and a Haar
    block of order `blk` on every run of blk rows, which spreads each row over all of them."""
    m, n = X.shape
    w = min(blk, m)
    q = m // w * w
    for _ in range(rounds):
        X = X[torch.randperm(m, generator=g, device=X.device)]
        H = torch.linalg.qr(torch.randn((w, w), generator=g, dtype=X.dtype, device=X.device))[0]
        X[:q] = torch.matmul(H, X[:q].reshape(q // w, w, n)).reshape(q, n)
    return X


def _ill_conditioned(m, n, k, seed):
    """Float32 A = U diag(s) V^T with s geometric from 1 to 1e-6, b = A x + 1e-10 noise (double)."""
    g = _gen(seed)
    s = torch.logspace(0, -6, n, dtype=torch.float64, device="cuda")
    R = _mix_rows(torch.eye(n, dtype=torch.float64, device="cuda"), g).t() * s[:, None]
    X = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    X[:n] = R
    A = tq.empty(m, n, dtype=torch.float32)
    A.copy_(_mix_rows(X, g))
    del X, R
    xt = torch.randn(n, k, generator=g, dtype=torch.float64, device="cuda")
    b = tq.empty(m, k)
    for r in range(0, m, 4096):
        b[r:r + 4096] = A[r:r + 4096].double() @ xt
    b += 1e-10 * torch.randn(m, k, generator=g, dtype=torch.float64, device="cuda")
    return A, b


def _batch_sizes(case):
    max_m = case["max_m"]
    return batched.random_sizes(case["nprob"], seed=case["nprob"] + max_m, max_m=max_m)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mixed":
        A, b = _ill_conditioned(case["m"], case["n"], case["k"], seed)
        return {"case": case, "A": A, "b": b}
    dtype = DTYPES[case["dtype"]]
    g = _gen(seed)
    if kind == "tile":
        nb, w, m2, ib = case["nb"], case["w"], case["m2"], min(case["ib"], case["nb"])
        shapes = {"A11": (nb, nb), "A12": (nb, w), "A21": (m2, nb), "A22": (m2, w)}
        orig = {k: _matrix(*s, dtype, g) for k, s in shapes.items()}
        return {"case": case, "ib": ib, "orig": orig, "work": {k: tq.empty(*s, dtype=dtype) for k, s in shapes.items()},
                "T1": tq.zeros(ib, nb, dtype=dtype), "T2": tq.zeros(ib, nb, dtype=dtype),
                "tau1": torch.zeros(nb, dtype=dtype, device="cuda"), "tau2": torch.zeros(nb, dtype=dtype, device="cuda")}
    if kind == "qr":
        m, n = case["m"], case["n"]
        ts, taus = tq.tile_shapes(m, n, case["nb"], case["ib"])
        return {"case": case, "A0": _matrix(m, n, dtype, g), "A": tq.empty(m, n, dtype=dtype),
                "T": tq.zeros(*ts, dtype=dtype), "tau": tq.zeros(*taus, dtype=dtype),
                "B0": _matrix(m, case["rhs"], dtype, g) if case["rhs"] else None,
                "B": tq.empty(m, case["rhs"], dtype=dtype) if case["rhs"] else None}
    if kind == "tall":
        m, n = case["m"], case["n"]
        return {"case": case, "A0": _matrix(m, n, dtype, g), "A": tq.empty(m, n, dtype=dtype)}
    if kind == "batched":
        bg = batched.BatchedGels(*_batch_sizes(case), dtype=dtype)
        A0, B0 = _batch_inputs(bg, dtype, g)
        return {"case": case, "bg": bg, "A0": A0, "B0": B0}
    A = _randn((case["batch"], case["m"], case["n"]), dtype, g).requires_grad_(True)
    dQ = _randn((case["batch"], case["m"], case["n"]), dtype, g)
    dR = torch.triu(_randn((case["batch"], case["n"], case["n"]), dtype, g))
    return {"case": case, "A": A, "dQ": dQ, "dR": dR}


def _batch_inputs(bg, dtype, g):
    """N(0, 1) problems with 3 sqrt(m) added on their diagonals: nearly square ones are then as well
    conditioned as a regularised fit, and X is as accurate as the element type allows."""
    A0 = torch.randn(bg.A.shape, generator=g, device="cuda", dtype=torch.float64)
    m, n = bg.desc["m"].astype(np.int64), bg.desc["n"].astype(np.int64)
    i = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n)              # 0 .. n_q - 1 of every problem
    at = torch.from_numpy(np.repeat(bg.desc["a_off"], n) + i * np.repeat(m + 1, n)).to("cuda")
    A0[at] += torch.from_numpy(np.repeat(3.0 * np.sqrt(m), n)).to("cuda")
    B0 = torch.randn(bg.B.shape, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    return A0.to(dtype), B0


# ---- one pass ---------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "tile":
        w = s["work"]
        for k, t in s["orig"].items():
            w[k].copy_(t)
        nb, m2, nw, ib = case["nb"], case["m2"], case["w"], s["ib"]
        tq.geqrt(nb, nb, ib, w["A11"], s["T1"], s["tau1"], None)
        tq.unmqr("L", "C", nb, nw, nb, ib, w["A11"], nb, s["T1"], w["A12"], None)
        tq.tsqrt(m2, nb, ib, w["A11"], w["A21"], s["T2"], s["tau2"], None)
        tq.tsmqr("L", "C", nb, nw, m2, nw, nb, ib, w["A12"], w["A22"], w["A21"], s["T2"], None)
        return [w["A11"], w["A12"], w["A21"], w["A22"], s["T1"], s["T2"], s["tau1"], s["tau2"]]
    if kind == "qr":
        s["A"].copy_(s["A0"])
        T, tau = tq.tile_geqrf(s["A"], case["nb"], case["ib"], T=s["T"], tau=s["tau"])
        out = [s["A"], T, tau]
        if s["B"] is not None:
            s["B"].copy_(s["B0"])
            tq.tile_unmqr("C", s["A"], T, s["B"], case["nb"], case["ib"])
            out.append(s["B"])
        return out
    if kind == "tall":
        s["A"].copy_(s["A0"])
        return [s["A"], *tq.tile_geqrf_tree(s["A"], case["nb"], case["ib"], grp=case["grp"])]
    if kind == "mixed":
        return tq.lstsq_mixed(s["A"], s["b"], case["nb"], case["ib"])[0]
    if kind == "batched":
        bg = s["bg"]
        bg.A.copy_(s["A0"])
        bg.B.copy_(s["B0"])
        bg.replay()
        return [bg.A, bg.B]
    Q, R = autodiff.qr(s["A"])
    (grad,) = torch.autograd.grad((Q, R), (s["A"],), (s["dQ"], s["dR"]))
    return [Q.detach(), R.detach(), grad]


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "mixed":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * m * n + 8 * (m + n) * k, "flops": 2 * m * n * n - 2 * n ** 3 / 3 + 4 * m * n * k}
    size = {"f64": 8, "f32": 4, "c128": 16}[case["dtype"]]
    mul = 4 if case["dtype"] == "c128" else 1
    if kind == "tile":
        nb, w, m2, ib = case["nb"], case["w"], case["m2"], min(case["ib"], case["nb"])
        elems = 2 * (nb * nb + nb * w + m2 * nb + m2 * w) + 2 * ib * nb + 2 * nb
        return {"bytes": size * elems,
                "flops": mul * (4 / 3 * nb ** 3 + 2 * nb * nb * w + 2 * m2 * nb * nb + 4 * m2 * nb * w)}
    if kind in ("qr", "tall"):
        m, n, nb, ib, rhs = case["m"], case["n"], case["nb"], case["ib"], case.get("rhs", 0)
        a, b = max(m, n), min(m, n)
        mt = -(-m // nb)
        return {"bytes": size * (2 * m * n + mt * ib * n + mt * n + 2 * m * rhs),
                "flops": mul * (2 * a * b * b - 2 * b ** 3 / 3 + rhs * (4 * m * b - 2 * b * b))}
    if kind == "batched":
        ms, ns, ks = (x.astype(np.float64) for x in _batch_sizes(case))
        return {"bytes": float(np.sum(2 * size * ms * (ns + ks))),
                "flops": float(np.sum(2 * ms * ns * ns - 2 * ns ** 3 / 3 + ks * (4 * ms * ns - ns * ns)))}
    b, m, n = case["batch"], case["m"], case["n"]
    # QR, forming Q, Q^T Qbar and Q X through the reflectors, the products and the triangular solve
    qr = 2 * m * n * n - 2 * n ** 3 / 3
    return {"bytes": size * b * (4 * m * n + 2 * n * n), "flops": b * (2 * qr + 2 * qr + 2 * m * n * n)}


# ---- the same results in 64 bits --------------------------------------------
# The tile algorithms column by column in plain torch (LAPACK's Householder convention: beta takes the
# sign opposite to the real part of alpha), on one matrix or on a stack of them.

MOST_STEPS = 60000       # column steps (about 0.2 ms each) beyond which exact() has no value


def _house(alpha, ss):
    """beta, tau, scale of the reflector for alpha over a vector of squared norm ss (stacks of scalars)."""
    a = alpha.real if alpha.is_complex() else alpha
    ai = alpha.imag if alpha.is_complex() else torch.zeros_like(a)
    beta = -torch.copysign(torch.sqrt(a * a + ai * ai + ss), a)
    zero = (ss == 0) & (ai == 0)
    safe = torch.where(zero, torch.ones_like(beta), beta)
    tau = (beta - a) / safe
    if alpha.is_complex():
        tau = torch.complex(tau, -ai / safe)
    one = torch.ones_like(alpha)
    scale = 1 / torch.where(zero, one, alpha - beta)
    return torch.where(zero, alpha, beta.to(alpha.dtype)), torch.where(zero, 0 * one, tau), torch.where(zero, 0 * one, scale)


def _cn(x):
    return x.mH if x.is_complex() else x.mT


def _block(rows, V, T):
    """rows := (I - V T V^H)^H rows; both are lists of row parts, rows' parts views that are updated."""
    W = sum(torch.matmul(_cn(v), c) for v, c in zip(V, rows))
    W = torch.matmul(_cn(T), W)
    for v, c in zip(V, rows):
        c -= torch.matmul(v, W)


def _geqrt(A, n, ib, T, tau):
    """geqrt on the first n columns of A (stack, m x N); the columns right of n are updated too."""
    m = A.shape[-2]
    k = min(m, n)
    for i0 in range(0, k, ib):
        sb = min(ib, k - i0)
        V = torch.zeros(A.shape[:-2] + (m - i0, sb), dtype=A.dtype, device=A.device)
        Tb = torch.zeros(A.shape[:-2] + (sb, sb), dtype=A.dtype, device=A.device)
        P = A[..., i0:, i0:min(i0 + ib, n)]
        for j in range(sb):
            x = P[..., j + 1:, j]
            if x.shape[-1] == 0:                          # a one-row column has no reflector
                V[..., j, j] = 1
                continue
            beta, t, sc = _house(P[..., j, j], (x.abs() ** 2).sum(-1))
            V[..., j, j] = 1
            V[..., j + 1:, j] = x * sc[..., None]
            v = V[..., :, j:j + 1]
            d = torch.matmul(_cn(v), P[..., j + 1:])
            P[..., j + 1:] -= v * (t.conj()[..., None, None] * d)
            P[..., j, j] = beta
            P[..., j + 1:, j] = v[..., j + 1:, 0]
            if j:
                Tb[..., :j, j:j + 1] = -t[..., None, None] * torch.matmul(Tb[..., :j, :j], torch.matmul(_cn(V[..., :j]), v))
            Tb[..., j, j] = t
            tau[..., i0 + j] = t
        T[..., :sb, i0:i0 + sb] = Tb
        if i0 + P.shape[-1] < A.shape[-1]:
            _block([A[..., i0:, i0 + P.shape[-1]:]], [V], Tb)


def _tsqrt(A1, A2, n, ib, T, tau, tri=False):
    """tsqrt of [upper A1; A2] over the first n columns, the columns right of n updated too.  tri: A2 is
    upper triangular there (ttqrt), entries below its diagonal belong to another factor and stay."""
    k = min(A1.shape[-2], n)
    if tri:
        k = min(k, A2.shape[-2])
    m2 = A2.shape[-2]
    X = torch.triu(A2[..., :, :n]) if tri else A2[..., :, :n]
    for i0 in range(0, k, ib):
        sb = min(ib, k - i0)
        e = min(i0 + ib, n)
        V2 = torch.zeros(A1.shape[:-2] + (m2, sb), dtype=A1.dtype, device=A1.device)
        Tb = torch.zeros(A1.shape[:-2] + (sb, sb), dtype=A1.dtype, device=A1.device)
        for j in range(sb):
            c = i0 + j
            x = X[..., :, c]
            beta, t, sc = _house(A1[..., c, c], (x.abs() ** 2).sum(-1))
            V2[..., :, j] = x * sc[..., None]
            v = V2[..., :, j:j + 1]
            d = t.conj()[..., None, None] * (A1[..., c:c + 1, c + 1:e] + torch.matmul(_cn(v), X[..., :, c + 1:e]))
            A1[..., c:c + 1, c + 1:e] -= d
            X[..., :, c + 1:e] -= v * d
            A1[..., c, c] = beta
            X[..., :, c] = v[..., :, 0]
            if j:
                Tb[..., :j, j:j + 1] = -t[..., None, None] * torch.matmul(Tb[..., :j, :j], torch.matmul(_cn(V2[..., :j]), v))
            Tb[..., j, j] = t
            tau[..., c] = t
        T[..., :sb, i0:i0 + sb] = Tb
        I1 = torch.eye(sb, dtype=A1.dtype, device=A1.device).expand(A1.shape[:-2] + (sb, sb))
        if e < n:                                         # the rest of the tile
            _block([A1[..., i0:i0 + sb, e:n], X[..., :, e:]], [I1, V2], Tb)
        if n < A1.shape[-1]:                              # the tile columns right of it
            _block([A1[..., i0:i0 + sb, n:], A2[..., :, n:]], [I1, V2], Tb)
    if tri:
        keep = torch.ones(m2, n, dtype=torch.bool, device=A1.device).triu()
        A2[..., :, :n] = torch.where(keep, X, A2[..., :, :n])


def _flat(A, nb, ib, n=None):
    """Flat-tree tile QR of the first n columns of A (stack) in place; T and tau in the library's layout."""
    m, n = A.shape[-2], n or A.shape[-1]
    mt, lead = -(-m // nb), A.shape[:-2]
    T = torch.zeros(lead + (mt * ib, n), dtype=A.dtype, device=A.device)
    tau = torch.zeros(lead + (n, mt), dtype=A.dtype, device=A.device)
    for k in range(-(-min(m, n) // nb)):
        c0, c1 = k * nb, min(n, (k + 1) * nb)
        top = A[..., k * nb:min(m, (k + 1) * nb), c0:]
        _geqrt(top, c1 - c0, ib, T[..., k * ib:(k + 1) * ib, c0:c1], tau[..., c0:c1, k])
        for i in range(k + 1, mt):
            _tsqrt(top, A[..., i * nb:min(m, (i + 1) * nb), c0:], c1 - c0, ib, T[..., i * ib:(i + 1) * ib, c0:c1],
                   tau[..., c0:c1, i])
    return T, tau


def _tree(A, nb, ib, grp):
    """The hierarchical form: groups of grp tiles flat into their first, those by a binary tree."""
    m, n = A.shape
    mt = -(-m // nb)
    out = [torch.zeros(s, dtype=A.dtype, device=A.device) for s in ((mt * ib, n), (n, mt), (mt * ib, n), (n, mt))]
    T, tau, T2, tau2 = out
    for k in range(-(-min(m, n) // nb)):
        c0, c1 = k * nb, min(n, (k + 1) * nb)
        w = c1 - c0

        def tile(i):
            return A[i * nb:min(m, (i + 1) * nb), c0:]

        def merge(i, p, tri):
            _tsqrt(tile(i), tile(p), w, ib, T2[p * ib:(p + 1) * ib, c0:c1], tau2[c0:c1, p], tri)

        ragged = mt - 1 > k and m - (mt - 1) * nb < w     # too few rows for a triangle: merged whole
        end = mt - 1 if ragged else mt
        leaders = list(range(k, end, grp))
        for i in leaders:
            _geqrt(tile(i), w, ib, T[i * ib:(i + 1) * ib, c0:c1], tau[c0:c1, i])
            for p in range(i + 1, min(i + grp, end)):
                merge(i, p, False)
        if ragged:
            merge(leaders[-1], mt - 1, False)
        s = grp
        while k + s < end:
            for i in range(k, end - s, 2 * s):
                merge(i, i + s, True)
            s *= 2
    return out


def _steps(case):
    nb = case.get("nb", 256)
    mt, kt = -(-case["m"] // nb), -(-min(case["m"], case["n"]) // nb)
    return sum(2 * (mt - k) if case["kind"] == "tall" else mt - k for k in range(kt)) * min(nb, case["n"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "mixed":
        A, b = _ill_conditioned(case["m"], case["n"], case["k"], seed)
        A = A.double()
        Q, R = torch.linalg.qr(A)
        x = torch.linalg.solve_triangular(R, Q.mT @ b, upper=True)
        for _ in range(2):
            x = x + torch.linalg.solve_triangular(R, Q.mT @ (b - A @ x), upper=True)
        return x
    dtype = DTYPES[case["dtype"]]
    wide = torch.complex128 if dtype.is_complex else torch.float64
    g = _gen(seed)
    if kind == "tile":
        nb, w, m2, ib = case["nb"], case["w"], case["m2"], min(case["ib"], case["nb"])
        A11, A12, A21, A22 = (_matrix(*s, dtype, g).to(wide) for s in ((nb, nb), (nb, w), (m2, nb), (m2, w)))
        top, low = torch.cat((A11, A12), 1), torch.cat((A21, A22), 1)
        T = [torch.zeros(ib, nb, dtype=wide, device="cuda") for _ in range(2)]
        tau = [torch.zeros(nb, dtype=wide, device="cuda") for _ in range(2)]
        _geqrt(top, nb, ib, T[0], tau[0])
        _tsqrt(top, low, nb, ib, T[1], tau[1])
        return [top[:, :nb], top[:, nb:], low[:, :nb], low[:, nb:], T[0], T[1], tau[0], tau[1]]
    if kind == "qr":
        if _steps(case) > MOST_STEPS:
            return None
        A = _matrix(case["m"], case["n"], dtype, g).to(wide)
        n = A.shape[1]
        if case["rhs"]:
            A = torch.cat((A, _matrix(case["m"], case["rhs"], dtype, g).to(wide)), 1)
        if case["rhs"] and n > case["m"]:                 # Q^H B needs the reflectors of the leading columns only
            F = A[:, :n].contiguous()
            T, tau = _flat(F, case["nb"], case["ib"])
            G = torch.cat((A[:, :case["m"]], A[:, n:]), 1)
            _flat(G, case["nb"], case["ib"], case["m"])
            return [F, T, tau, G[:, case["m"]:]]
        T, tau = _flat(A, case["nb"], case["ib"], n)
        return [A[:, :n], T, tau] + ([A[:, n:]] if case["rhs"] else [])
    if kind == "tall":
        if _steps(case) > MOST_STEPS:
            return None
        A = _matrix(case["m"], case["n"], dtype, g).to(wide)
        return [A, *_tree(A, case["nb"], case["ib"], case["grp"])]
    if kind == "batched":
        bg = batched.BatchedGels(*_batch_sizes(case), dtype=dtype)      # the plan's offsets only
        A0, B0 = _batch_inputs(bg, dtype, g)
        A, B = A0.double().cpu(), B0.double().cpu()
        for q in range(bg.nprob):
            a, b = bg.a_view(q, A), bg.b_view(q, B)
            h, tau = torch.geqrf(a)
            y = torch.ormqr(h, tau, b, left=True, transpose=True)
            n = h.shape[1]
            y[:n] = torch.linalg.solve_triangular(h[:n].triu(), y[:n], upper=True)
            a.copy_(h)
            b.copy_(y)
        return [A, B]
    A = _randn((case["batch"], case["m"], case["n"]), dtype, g)
    dQ = _randn((case["batch"], case["m"], case["n"]), dtype, g)
    dR = torch.triu(_randn((case["batch"], case["n"], case["n"]), dtype, g))
    F = A.clone()
    _flat(F, 256, 32)
    R = torch.triu(F[:, :case["n"]])
    Q = torch.linalg.qr(A)[0]                             # its columns up to their signs, which R's rows give
    Q = Q * torch.sign((Q.mT @ A).diagonal(dim1=1, dim2=2) * R.diagonal(dim1=1, dim2=2))[:, None, :]
    M = R @ dR.mT - dQ.mT @ Q
    M = torch.tril(M) + torch.tril(M, -1).mT
    grad = torch.linalg.solve_triangular(R.mT, dQ + Q @ M, upper=False, left=False)
    return [Q, R, grad]
