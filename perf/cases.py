"""The calls whose speed counts: whole solves, solves on a resident factor, Kalman smoothing,
batches of uneven systems and bursts of served requests, each through the package's public API.

``listed()`` holds the fixed cases, ``draw(rng)`` gives others of the same ranges; a case is
prepared (``prepare``: seeded inputs and the handle), run (``run``: one pass) and has a bound on
its work (``work``) and a 64-bit answer made without the package (``exact``).
"""
import math

import numpy as np
import torch

import blockstructuredsolvers_gb300 as bss

KF_SIZES = (8, 16, 32, 64)
BATCH_SIZES = (16, 32, 48, 64, 96, 128)


def listed():
    return [
        # The reference's own test and example size in its default type: one small system, factored
        # and solved in place; latency and launches are all of it.
        {"name": "f64_small", "kind": "solve", "N": 100, "n": 32, "k": 1, "T": "f64", "precision": "plain"},
        # An ordinary system of an odd block size and an odd number of right-hand sides.
        {"name": "f64_ragged", "kind": "solve", "N": 1531, "n": 37, "k": 3, "T": "f64", "precision": "plain"},
        # The large system in plain FP64: what a user of the reference runs unchanged.
        {"name": "f64_large", "kind": "solve", "N": 16384, "n": 64, "k": 1, "T": "f64", "precision": "plain"},
        # Wide blocks in plain FP64 (an optimal-control problem with many states per stage).
        {"name": "f64_wide", "kind": "solve", "N": 2048, "n": 128, "k": 4, "T": "f64", "precision": "plain"},
        # The large system in plain FP32 with a block of right-hand sides.
        {"name": "f32_large_k16", "kind": "solve", "N": 16384, "n": 64, "k": 16, "T": "f32", "precision": "plain"},
        # The headline: FP32 factors refined to FP64 accuracy.
        {"name": "mixed_large", "kind": "solve", "N": 16384, "n": 64, "k": 1, "T": "f64", "precision": "mixed"},
        # The largest system: log-spaced spectra over [1, 1e4], four right-hand sides, refined.
        {"name": "mixed_wide", "kind": "solve", "N": 65536, "n": 128, "k": 4, "T": "f64", "precision": "mixed"},
        # New right-hand sides on a resident factor: many columns, refined.
        {"name": "rhs_mixed_k16", "kind": "rhs", "N": 16384, "n": 64, "k": 16, "T": "f64", "precision": "mixed"},
        # New right-hand side on a resident factor of small blocks: the inner step of a control loop.
        {"name": "rhs_f64_small", "kind": "rhs", "N": 2000, "n": 16, "k": 1, "T": "f64", "precision": "plain"},
        # One Kalman smoother: blocks built from the model on the device, factored and solved.
        {"name": "kalman_n16", "kind": "kalman", "N": 5000, "n": 16, "k": 1, "T": "f64", "precision": "mixed"},
        # Many uneven systems in one batch.
        {"name": "batch_64", "kind": "batch", "S": 64, "Nmax": 1024, "T": "f64", "precision": "mixed"},
        # A burst of Kalman requests at the server, from host buffers to host buffers, 30% of them
        # new observations on a resident factor.
        {"name": "served_48", "kind": "served", "S": 48, "Nmax": 5000, "T": "f64", "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("solve",) * 6 + ("rhs",) * 2 + ("kalman", "batch", "served"))
    if kind == "kalman":
        return {"kind": kind, "N": _log_int(rng, 50, 5000), "n": rng.choice(KF_SIZES + (12, 27)), "k": rng.choice((1, 1, 2)),
                "T": "f64", "precision": rng.choice(("mixed", "mixed", "plain"))}
    if kind == "batch":
        return {"kind": kind, "S": rng.randint(8, 64), "Nmax": rng.randint(64, 1024), "T": "f64", "precision": "mixed"}
    if kind == "served":
        return {"kind": kind, "S": rng.randint(8, 48), "Nmax": rng.randint(500, 5000), "T": "f64", "precision": "mixed"}
    T, precision = rng.choice((("f64", "plain"), ("f64", "plain"), ("f32", "plain"), ("f64", "mixed"), ("f64", "mixed")))
    # block sizes: the usual powers of two as often as any other
    n = rng.choice((8, 16, 32, 64, 128)) if rng.random() < 0.4 else _log_int(rng, 4, 128)
    k = rng.choice((1, 1, 1, 2, 3, 4, 8, 16))
    # FP64 products cost about sixty times FP32's: no more of either than the largest listed case has
    most = 4.5e9 if (T, precision) == ("f64", "plain") else 1.3e11
    top = min(65536, most / n**3, 4e9 / (n * n * max(k, 4)))
    return {"kind": kind, "N": _log_int(rng, 16, max(16, int(top))), "n": n, "k": k, "T": T, "precision": precision}


# ---------------------------------------------------------------------------------------------
# inputs: blocks (N, n, n), right-hand sides (N, n, k), FP64 on the GPU
# ---------------------------------------------------------------------------------------------
def _orthogonal(g, count, n):
    Q, R = torch.linalg.qr(torch.randn((count, n, n), dtype=torch.float64, device="cuda", generator=g))
    s = torch.where(torch.diagonal(R, dim1=1, dim2=2) < 0, -1.0, 1.0).to(torch.float64)
    return Q * s[:, None, :]


def _log_spectrum(g, N, n, k):
    """A_i = Q_i diag(lambda) Q_i^T with lambda log-spaced over [1, 1e4] and B_i = 0.45 U_i V_i^T;
    each orthogonal factor is a product of two drawn from a pool."""
    lam = torch.logspace(0, 4, n, dtype=torch.float64, device="cuda")
    pool = _orthogonal(g, 64, n)
    pick = lambda c: pool[torch.randint(0, 64, (c,), device="cuda", generator=g)]
    A = torch.empty((N, n, n), dtype=torch.float64, device="cuda")
    B = torch.empty((N - 1, n, n), dtype=torch.float64, device="cuda")
    for s in range(0, N, 8192):
        c = min(8192, N - s)
        Q = pick(c) @ pick(c)
        M = (Q * lam) @ Q.mT
        A[s:s + c] = 0.5 * (M + M.mT)
    for s in range(0, N - 1, 8192):
        c = min(8192, N - 1 - s)
        B[s:s + c] = 0.45 * (pick(c) @ pick(c).mT)
    return A, B, torch.randn((N, n, k), dtype=torch.float64, device="cuda", generator=g)


def _shifted(g, N, n, k, shift, b_scale):
    """A_i = G G^T + shift I, B_i = b_scale N(0, 1), d ~ U[0, 1)."""
    A = torch.empty((N, n, n), dtype=torch.float64, device="cuda")
    for s in range(0, N, 8192):
        G = torch.randn((min(8192, N - s), n, n), dtype=torch.float64, device="cuda", generator=g)
        A[s:s + G.shape[0]] = G @ G.mT
    A.diagonal(dim1=1, dim2=2).add_(shift)
    B = torch.randn((max(N - 1, 0), n, n), dtype=torch.float64, device="cuda", generator=g).mul_(b_scale)
    return A, B, torch.rand((N, n, k), dtype=torch.float64, device="cuda", generator=g)


def _system(case, seed):
    """The system of a "solve" or "rhs" case, rounded to its type."""
    N, n, k = case["N"], case["n"], case["k"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if n > 64 and case["precision"] == "mixed":
        S = _log_spectrum(g, N, n, k)
    elif n >= 32:  # the reference tests' family: diagonally dominant enough for n > 16
        S = _shifted(g, N, n, k, float(n), 1.0)
    else:
        S = _shifted(g, N, n, k, 2.0 * n, 0.5)
    return [t.to(torch.float32 if case["T"] == "f32" else torch.float64) for t in S]


def _batch_shapes(case, seed):
    """Sizes of a batch's systems: they go with the case, and not with the seed."""
    r = np.random.default_rng(1000 * case["S"] + case["Nmax"])
    S = case["S"]
    return (r.integers(16, case["Nmax"] + 1, S).tolist(), r.choice(BATCH_SIZES, S).tolist(), r.integers(1, 9, S).tolist())


def _kalman_model(r, n):
    m = n // 2
    F = r.standard_normal((n, n))
    F *= 0.95 / np.abs(np.linalg.eigvals(F)).max()
    return F, r.standard_normal((m, n)), 10.0 * np.eye(n), 2.0 * np.eye(m)


def _observations(r, F, H, N, k):
    """k observation sequences simulated from the model, (N, k, m)."""
    n, m = F.shape[0], H.shape[0]
    W = math.sqrt(0.1) * r.standard_normal((N, k, n))
    X, x, Ft = np.empty((N, k, n)), np.zeros((k, n)), np.ascontiguousarray(F.T)
    for t in range(N):
        x = x @ Ft + W[t]
        X[t] = x
    return X @ H.T + math.sqrt(0.5) * r.standard_normal((N, k, m))


def _served_requests(case, seed):
    """(models, requests): a request is (model, horizon, observations, is a new model). Sizes go
    with the case, values with the seed."""
    shape, r = np.random.default_rng(1000 * case["S"] + case["Nmax"]), np.random.default_rng(seed)
    models, reqs = [], []
    for _ in range(case["S"]):
        new = not models or shape.random() >= 0.3
        if new:
            models.append((_kalman_model(r, int(shape.choice(KF_SIZES))), int(shape.integers(50, case["Nmax"] + 1))))
        a = len(models) - 1 if new else int(shape.integers(0, len(models)))
        (F, H, _, _), N = models[a]
        reqs.append((a, N, _observations(r, F, H, N, 1), new))
    return models, reqs


def _blocks(t):
    """(N, a, b) blocks as the (a, b, N) column-major tensor that the package's tensors are."""
    return t.mT.contiguous().permute(2, 1, 0)


def _dtype(case):
    return torch.float32 if case["T"] == "f32" else torch.float64


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "rhs"):
        N, n, k = case["N"], case["n"], case["k"]
        A, B, d = (_blocks(t) for t in _system(case, seed))
        data = bss.initialize_batched(N, n, _dtype(case), k=k, precision=case["precision"])
        s = {"kind": kind, "data": data, "d": d, "x": data.d_tensor[:, :, :N]}
        if kind == "solve" and case["precision"] == "plain":  # factored in place: each pass brings its blocks
            s.update(A=A, B=B, A_in=data.A_tensor[:, :, :N], B_in=data.B_tensor[:, :, :N - 1])
        else:
            data.A_tensor[:, :, :N].copy_(A)
            data.B_tensor[:, :, :N - 1].copy_(B)
        if kind == "rhs":
            bss.factorize_(data)
        return s
    if kind == "kalman":
        N, n, k = case["N"], case["n"], case["k"]
        r = np.random.default_rng(seed)
        F, H, Qi, Ri = _kalman_model(r, n)
        y = torch.from_numpy(_observations(r, F, H, N, k)).cuda().permute(2, 1, 0)
        dev = [torch.from_numpy(np.ascontiguousarray(M.T)).cuda().T for M in (F, H, Qi, Ri)]
        data = bss.initialize_batched(N, n, torch.float64, k=k, precision=case["precision"])
        return {"kind": kind, "data": data, "model": dev, "y": y, "x": data.d_tensor[:, :, :N]}
    if kind == "batch":
        Ns, ns, ks = _batch_shapes(case, seed)
        b = bss.initialize_multi(Ns, ns, ks, torch.float64, precision=case["precision"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        ds = []
        for sv in b.systems:
            A, B, d = (_blocks(t) for t in _shifted(g, sv.N, sv.n, sv.k, 2.0 * sv.n, 0.5))
            sv.A_tensor.copy_(A)
            sv.B_tensor.copy_(B)
            ds.append(d)
        return {"kind": kind, "batch": b, "d": ds, "x": [sv.d_tensor for sv in b.systems]}
    models, reqs = _served_requests(case, seed)
    pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
    models = [[pin(M.T) for M in mats] for mats, _ in models]
    reqs = [(a, pin(y), torch.empty((N, 1, models[a][0].shape[0]), dtype=torch.float64, pin_memory=True), new)
            for a, N, y, new in reqs]
    return {"kind": kind, "server": bss.Server(precision=case["precision"]), "models": models, "reqs": reqs}


def run(state):
    kind = state["kind"]
    if kind in ("solve", "rhs"):
        data = state["data"]
        if "A" in state:
            state["A_in"].copy_(state["A"])
            state["B_in"].copy_(state["B"])
        state["x"].copy_(state["d"])
        if kind == "solve":
            bss.factorize_(data)
        bss.solve_(data)
        return state["x"]
    if kind == "kalman":
        data = state["data"]
        F, H, Qi, Ri = state["model"]
        bss.kf_build(F, H, Qi, Ri, state["y"], data.A_tensor, data.B_tensor, data.d_tensor)
        bss.factorize_(data)
        bss.solve_(data)
        return state["x"]
    if kind == "batch":
        b = state["batch"]
        for x, d in zip(state["x"], state["d"]):
            x.copy_(d)
        b.factorize()
        b.solve()
        return state["x"]
    srv, factors, ids = state["server"], {}, []
    for a, y, x, new in state["reqs"]:
        if new:
            rid, factors[a] = srv.submit_kalman(*state["models"][a], y, x, keep=True)
        else:
            rid = srv.submit_rhs(factors[a], y, x)
        ids.append(rid)
    for rid in ids:
        srv.wait(rid)
    for f in factors.values():
        srv.release(f)
    return [x for _, _, x, _ in state["reqs"]]


def work(case):
    """Flops of a sequential block Cholesky and its solves; bytes of the inputs and the outputs."""
    kind = case["kind"]
    if kind == "batch":
        systems = [(N, n, k, (2 * N - 1) * n * n + 2 * N * n * k) for N, n, k in zip(*_batch_shapes(case, 0))]
    elif kind == "served":
        models, reqs = _served_requests(case, 0)
        systems = [(N, H.shape[1], 1 if new else -1, N * sum(H.shape)) for a, N, _, new in reqs for H in (models[a][0][1],)]
    else:
        N, n, k = case["N"], case["n"], case["k"]
        values = N * k * (n + n // 2) if kind == "kalman" else (2 * N - 1) * n * n + 2 * N * n * k
        systems = [(N, n, -k if kind == "rhs" else k, values)]
    flops = values = 0
    for N, n, k, v in systems:  # k < 0: on a resident factor
        flops += (N * n**3 / 3 + 2 * (N - 1) * n**3 if k > 0 else 0) + abs(k) * (6 * N - 4) * n * n
        values += v
    return {"bytes": values * (4 if case["T"] == "f32" else 8), "flops": flops}


# ---------------------------------------------------------------------------------------------
# 64-bit answers: cyclic reduction in torch, refined once
# ---------------------------------------------------------------------------------------------
def _reduce(A, B, d):
    N = A.shape[0]
    if N == 1:
        return torch.cholesky_solve(d, torch.linalg.cholesky(A))
    n, k = A.shape[1], d.shape[2]
    odd = N // 2  # blocks 1, 3, ... are eliminated; each has a left neighbour, all but perhaps the last a right one
    right = (N - 1) // 2
    L = torch.linalg.cholesky(A[1::2])
    left_B, right_B = B[0::2], B[1::2]
    R = torch.zeros((odd, n, 2 * n + k), dtype=A.dtype, device=A.device)
    R[:, :, :n] = left_B.mT
    R[:right, :, n:2 * n] = right_B
    R[:, :, 2 * n:] = d[1::2]
    R = torch.cholesky_solve(R, L)
    A2, d2 = A[0::2].clone(), d[0::2].clone()
    A2[:odd] -= left_B @ R[:, :, :n]
    d2[:odd] -= left_B @ R[:, :, 2 * n:]
    A2[1:1 + right] -= right_B.mT @ R[:right, :, n:2 * n]
    d2[1:1 + right] -= right_B.mT @ R[:right, :, 2 * n:]
    B2 = -(left_B[:right] @ R[:right, :, n:2 * n])
    xe = _reduce(0.5 * (A2 + A2.mT), B2[:A2.shape[0] - 1], d2)
    x = torch.empty_like(d)
    x[0::2] = xe
    xo = R[:, :, 2 * n:] - R[:, :, :n] @ xe[:odd]
    xo[:right] -= R[:right, :, n:2 * n] @ xe[1:1 + right]
    x[1::2] = xo
    return x


def _solve64(A, B, d):
    A, B, d = A.double(), B.double(), d.double()
    x = _reduce(A, B, d)
    r = d - A @ x
    r[:-1] -= B @ x[1:]
    r[1:] -= B.mT @ x[:-1]
    return x + _reduce(A, B, r)


def _kalman64(mats, y):
    """The smoother's solution (N, n, k) for observations y (N, k, m)."""
    F, H, Qi, Ri = (torch.from_numpy(M).cuda() for M in mats)
    y = torch.from_numpy(y).cuda()
    N, n = y.shape[0], F.shape[0]
    A = (H.T @ Ri @ H + Qi + F.T @ Qi @ F).expand(N, n, n)
    return _solve64(A, (-(F.T @ Qi)).expand(N - 1, n, n), (y @ (Ri @ H)).mT)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "rhs"):
        return _blocks(_solve64(*_system(case, seed)))
    if kind == "kalman":
        r = np.random.default_rng(seed)
        mats = _kalman_model(r, case["n"])
        return _blocks(_kalman64(mats, _observations(r, mats[0], mats[1], case["N"], case["k"])))
    if kind == "batch":
        g = torch.Generator(device="cuda").manual_seed(seed)
        return [_blocks(_solve64(*_shifted(g, N, n, k, 2.0 * n, 0.5))) for N, n, k in zip(*_batch_shapes(case, seed))]
    models, reqs = _served_requests(case, seed)
    return [_kalman64(models[a][0], y).mT.contiguous() for a, _, y, _ in reqs]
