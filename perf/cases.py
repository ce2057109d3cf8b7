"""Performance cases of the framework's public entry points.

Each case is one thing that a user's program does over and over: a small
``solve``, a step sequence of a batch of independent instances, a pass over a
large data stream, a step of one large Burgers instance, a gradient sweep.

``listed`` names the cases, ``draw`` makes one more of the same ranges,
``prepare`` makes a case's inputs and handles from a seed, ``run`` is one pass
through the entry points, ``work`` what a pass cannot do without, and
``exact`` the same results from plain 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from __graft_entry__ import load_package

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: a user's first solve of a tiny Sylvester problem, every step kept
        dict(name="solve_small", kind="solve", n=40, m=36, r=4, nsub=2, steps=5, dt=1e-2, keep=True),
        # one stiff diffusion problem on a 256 x 256 grid (FP64, RK4 with 20 substeps), final state only
        dict(name="solve_laplace_256", kind="laplace", n=256, r=8, nsub=20, steps=20),
        # compression of a short recorded data stream (the reference's 100 x 100 rotation), every step kept
        dict(name="solve_data_100", kind="data", n=100, r=12, steps=10),
        # parameter study, FP32: many uneven Lyapunov problems advanced together
        dict(name="ensemble_fp32", kind="ensemble", alg="bug", precision="fp32", count=2048, nmin=64, nmax=1024,
             rmin=4, rmax=32, steps=4),
        # parameter study on one grid with graded cores: well-conditioned members in FP32, the others in double-float
        dict(name="ensemble_mixed", kind="mixed", n=256, m=256, count=1024, rmin=4, rmax=32, steps=4),
        # the plain FP64 form of a moderate uneven ensemble
        dict(name="ensemble_fp64", kind="ensemble", alg="bug", precision="fp64", count=512, nmin=64, nmax=1024,
             rmin=4, rmax=32, steps=2),
        # rank-adaptive ensemble on one grid (FP32)
        dict(name="ensemble_adaptive", kind="adaptive", precision="fp32", n=192, m=160, count=512, r=8, rcap=16,
             steps=3),
        # the data-compression stream: 8192 x 4096 snapshots, rank 64, rank-adaptive
        dict(name="stream_8192x4096", kind="stream", n=8192, m=4096, K=64, rmax=96, snaps=3),
        # a small stream of odd shape
        dict(name="stream_1001x517", kind="stream", n=1001, m=517, K=24, rmax=48, snaps=3),
        # Burgers uncertainty quantification, 4096 grid points x 16384 samples, at the rank it starts with
        dict(name="burgers_rank16", kind="burgers", n=4096, m=16384, r=16, nsub=64),
        # the same at the upper end of its rank range
        dict(name="burgers_rank64", kind="burgers", n=4096, m=16384, r=64, nsub=64),
        # loss and gradient through a few steps of the 2048 x 2048 problem (forward and backward)
        dict(name="gradient_2048", kind="gradient", n=2048, m=2048, r=32, rt=40, steps=4, every=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "laplace", "data", "ensemble", "ensemble", "mixed", "adaptive", "stream", "burgers",
                       "gradient"])
    if kind == "solve":
        n, m = _log(rng, 24, 200), _log(rng, 24, 200)
        return dict(kind=kind, n=n, m=m, r=rng.randint(2, 8), nsub=rng.randint(1, 3), steps=rng.randint(3, 8),
                    dt=1e-2, keep=rng.random() < 0.5)
    if kind == "laplace":
        return dict(kind=kind, n=rng.randint(100, 256), r=rng.randint(4, 8), nsub=20, steps=rng.randint(8, 20))
    if kind == "data":
        return dict(kind=kind, n=rng.randint(60, 160), r=rng.randint(4, 12), steps=rng.randint(5, 12))
    if kind == "ensemble":
        prec = rng.choice(["fp32", "df", "fp64"])
        most = {"fp32": 2048, "df": 768, "fp64": 384}[prec]
        rmin = rng.randint(3, 8)
        return dict(kind=kind, alg=rng.choice(["bug", "bug", "ksl"]), precision=prec,
                    count=_log(rng, 16, most), nmin=rng.randint(48, 128), nmax=rng.randint(256, 1024), rmin=rmin,
                    rmax=rmin + rng.randint(4, 24), steps=rng.randint(1, 3))
    if kind == "mixed":
        return dict(kind=kind, n=rng.randint(96, 384), m=rng.randint(96, 384), count=_log(rng, 64, 768),
                    rmin=rng.randint(4, 8), rmax=rng.randint(24, 32), steps=rng.randint(1, 4))
    if kind == "adaptive":
        r = rng.randint(3, 10)
        return dict(kind=kind, precision=rng.choice(["fp32", "fp64"]), n=rng.randint(64, 256), m=rng.randint(64, 256),
                    count=_log(rng, 32, 384), r=r, rcap=r + rng.randint(4, 8), steps=rng.randint(1, 3))
    if kind == "stream":
        K = rng.randint(12, 64)
        return dict(kind=kind, n=_log(rng, 512, 8192), m=_log(rng, 384, 4096), K=K, rmax=min(96, K + rng.randint(8, 32)),
                    snaps=3)
    if kind == "burgers":
        return dict(kind=kind, n=256 * rng.randint(1, 12), m=_log(rng, 512, 12000), r=rng.randint(8, 60),
                    nsub=rng.randint(24, 48))
    return dict(kind=kind, n=_log(rng, 128, 1800), m=_log(rng, 128, 1800), r=rng.randint(6, 32), rt=40,
                steps=rng.randint(2, 4), every=rng.randint(1, 3))


# ---------------------------------------------------------------------------
# Inputs (made from the seed alone)
# ---------------------------------------------------------------------------

def _gen(seed, device=DEV):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _orthonormal(g, n, r, nmax, rmax):
    """Orthonormal factors of many members, zero padded to nmax x rmax (n, r: sizes per member)."""
    cnt = len(n)
    rows = torch.arange(nmax, device=DEV)[None, :] < n[:, None]
    cols = torch.arange(rmax, device=DEV)[None, :] < r[:, None]
    mask = (rows[:, :, None] & cols[:, None, :]).to(F64)
    X = torch.randn((cnt, nmax, rmax), generator=g, device=DEV, dtype=F64) * mask
    fill = torch.diag_embed((~cols).to(F64))
    for _ in range(2):
        L = torch.linalg.cholesky(X.transpose(1, 2) @ X + fill)
        X = torch.linalg.solve_triangular(L.transpose(1, 2), X, upper=True, left=False) * mask
    return X, rows, cols


def _tridiagonal(g, rows):
    """Stable tridiagonal operators: off-diagonals U[0.5, 1], diagonal -2 - U[0, 1] (count x 3 x nmax)."""
    cnt, nmax = rows.shape
    u = torch.rand((cnt, 3, nmax), generator=g, device=DEV, dtype=F64)
    tri = torch.stack([0.5 + 0.5 * u[:, 0], -2.0 - u[:, 1], 0.5 + 0.5 * u[:, 2]], dim=1)
    return tri * rows[:, None, :]


def _members(case, seed):
    """Padded factors and operators of an ensemble case, rounded to its storage type."""
    g = _gen(seed)
    cnt = case["count"]
    # a case has one set of sizes; the seed gives the members' data
    host = np.random.default_rng([cnt, case.get("nmin", 0), case.get("nmax", 0), case.get("rmax", 0)])
    if case["kind"] == "ensemble":
        n = host.integers(case["nmin"], case["nmax"] + 1, cnt)
        m = host.integers(case["nmin"], case["nmax"] + 1, cnt)
        r = host.integers(case["rmin"], case["rmax"] + 1, cnt)
        rate = 0.25
    else:
        n, m = np.full(cnt, case["n"]), np.full(cnt, case["m"])
        r = (np.full(cnt, case["r"]) if case["kind"] == "adaptive" else
             host.integers(case["rmin"], case["rmax"] + 1, cnt))
        rate = 1.0
    nt, mt, rt = (torch.from_numpy(x).to(DEV) for x in (n, m, r))
    U, rn, cols = _orthonormal(g, nt, rt, int(n.max()), int(r.max()))
    V, rm, _ = _orthonormal(g, mt, rt, int(m.max()), int(r.max()))
    k = torch.arange(1, int(r.max()) + 1, device=DEV, dtype=F64)
    S = torch.diag_embed(torch.exp2(-rate * k)[None, :] * cols)
    A, B = _tridiagonal(g, rn), _tridiagonal(g, rm)
    if case.get("precision") == "fp32":
        U, S, V, A, B = (x.float().double() for x in (U, S, V, A, B))
    return dict(n=n, m=m, r=r, U=U, S=S, V=V, A=A, B=B, rows=rn, cols_m=rm, cols=cols)


def _packed(X, keep):
    """Members' column-major blocks back to back (X: count x columns x rows, keep: which entries exist)."""
    return X[keep]


def _stream_parts(case, seed):
    """Modes and amplitudes of the rotating data stream sum_k sigma_k(t) u_k(t) v_k(t)^T."""
    g = _gen(seed)
    n, m, K = case["n"], case["m"], case["K"]
    sub = min(2 * K, n, m)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV, dtype=F64)  # noqa: E731
    Qu, Qv = torch.linalg.qr(rnd(n, sub))[0], torch.linalg.qr(rnd(m, sub))[0]
    Wu, Wv = (math.sqrt(0.1) * rnd(sub, sub) for _ in range(2))
    Wu, Wv = (torch.triu(W, 1) - torch.triu(W, 1).T for W in (Wu, Wv))
    f = 0.5 + 1.5 * torch.rand(K, generator=g, device=DEV, dtype=F64)
    k = torch.arange(1, K + 1, device=DEV, dtype=F64)
    noise = 1e-4 * torch.randn((m, n), generator=g, device=DEV, dtype=torch.float32)
    return Qu, Qv, Wu, Wv, f, k, noise


def _snapshots(case, seed):
    """Device snapshots (m x n row-major, which is n x m column-major) in FP32, and the rank-K factors at t = 0."""
    Qu, Qv, Wu, Wv, f, k, noise = _stream_parts(case, seed)
    K = case["K"]
    out = []
    for j in range(case["snaps"]):
        t = j / 499.0
        sig = torch.exp(-k / 8.0) * (1.0 + 0.3 * torch.sin(2 * math.pi * f * t))
        Ut = (Qu @ torch.linalg.matrix_exp(t * Wu))[:, :K] * sig
        Vt = (Qv @ torch.linalg.matrix_exp(t * Wv))[:, :K]
        out.append((Vt @ Ut.T + noise.double()).float())
    return out, (Qu[:, :K], torch.exp(-k / 8.0), Qv[:, :K])


def _burgers_parts(case, seed):
    """Viscous Burgers with random viscosity and second mode per sample (exact rank 3, completed to rank r)."""
    n, m, r = case["n"], case["m"], case["r"]
    g = np.random.default_rng(seed)
    x = np.arange(n) / n
    nu = g.uniform(0.005, 0.02, m)
    a, phi = g.uniform(0.0, 0.5, m), g.uniform(0.0, 2 * np.pi, m)
    B = np.stack([np.sin(2 * np.pi * x), np.sin(4 * np.pi * x), np.cos(4 * np.pi * x)], axis=1)
    C = np.stack([np.ones(m), a * np.cos(phi), a * np.sin(phi)], axis=1)
    Qb, Rb = np.linalg.qr(B)
    Qc, Rc = np.linalg.qr(C)
    P, s3, Qt = np.linalg.svd(Rb @ Rc.T)

    def complete(Q):
        Z = g.standard_normal((Q.shape[0], r - 3))
        for _ in range(2):
            Z -= Q @ (Q.T @ Z)
        return np.hstack([Q, np.linalg.qr(Z)[0]])

    U, V = complete(Qb @ P), complete(Qc @ Qt.T)
    s = np.concatenate([s3, np.zeros(r - 3)])
    f32 = lambda X: X.astype(np.float32).astype(np.float64)  # noqa: E731
    dt = min(1e-4, case["nsub"] * 2.1 / (4 * 0.02 * n * n))
    return f32(U), f32(s), f32(V), f32(nu), 1.0 / n, dt


def _laplace_parts(case, seed):
    n, r = case["n"], case["r"]
    g = np.random.default_rng(seed)
    h = 1.0 / (n + 1)
    A = (np.full(n, 1 / h**2), np.full(n, -2 / h**2 - 0.1), np.full(n, 1 / h**2))
    x = np.arange(1, n + 1) * h
    modes = np.sin(np.pi * np.outer(x, np.arange(1, 13)))
    # smooth initial data: the lowest 12 sine modes, mixed
    U, V = (np.linalg.qr(modes @ np.linalg.qr(g.standard_normal((12, r)))[0])[0] for _ in range(2))
    dt = 1e-4 * (257.0 * h) ** 2
    return A, U, np.diag(2.0 ** -np.arange(1, r + 1)), V, dt


def _solve_parts(case, seed):
    n, m, r = case["n"], case["m"], case["r"]
    g = np.random.default_rng(seed)
    A = (g.uniform(0.5, 1, n), -2 - g.uniform(0, 1, n), g.uniform(0.5, 1, n))
    B = (g.uniform(0.5, 1, m), -2 - g.uniform(0, 1, m), g.uniform(0.5, 1, m))
    U, V = np.linalg.qr(g.standard_normal((n, r)))[0], np.linalg.qr(g.standard_normal((m, r)))[0]
    return A, B, U, np.diag(2.0 ** -np.arange(1, r + 1)), V


def _data_parts(case, seed):
    """Y(t) = exp(t W1) e^t D exp(t W2) at steps of 0.01, and the truncated SVD of Y(0)."""
    N, r = case["n"], case["r"]
    g = np.random.default_rng(seed)
    W1, W2 = (torch.from_numpy(np.triu(W, 1) - np.triu(W, 1).T) for W in (g.standard_normal((N, N)) for _ in range(2)))
    D = torch.diag(torch.exp2(-torch.arange(1, N + 1, dtype=F64)))
    snaps = [(torch.linalg.matrix_exp(0.01 * j * W1) @ (math.exp(0.01 * j) * D)
              @ torch.linalg.matrix_exp(0.01 * j * W2)).numpy() for j in range(case["steps"] + 1)]
    return snaps, np.eye(N)[:, :r].copy(), np.diag(2.0 ** -np.arange(1, r + 1)), np.eye(N)[:, :r].copy()


def _gradient_parts(case, seed):
    n, m, r, rt = case["n"], case["m"], case["r"], case["rt"]
    g = np.random.default_rng(seed)
    A0 = (np.ones(n), -2.0 * np.ones(n), np.ones(n))
    B = (np.ones(m), -2.0 * np.ones(m), np.ones(m))
    theta = g.normal(0.0, math.sqrt(0.1), n)
    q = lambda a, b: np.linalg.qr(g.standard_normal((a, b)))[0]  # noqa: E731
    U, V, P, Q = q(n, r), q(m, r), q(n, rt), q(m, rt)
    return (A0, B, theta, U, np.diag(2.0 ** (-np.arange(1, r + 1) / 4.0)), V,
            P, np.diag(2.0 ** (-np.arange(1, rt + 1) / 4.0)), Q)


ENSEMBLE_DT = 1e-2


def _algorithm(lri, case):
    if case["kind"] == "adaptive":
        return lri.RankAdaptiveUnconventionalAlgorithm(1e-6, rmax=case["rcap"], K_alg=lri.RK4(1))
    if case.get("alg") == "ksl":
        return lri.ProjectorSplitting(lri.Strang(), lri.RK4(1))
    return lri.UnconventionalAlgorithm(lri.RK4(1))


def prepare(case, seed):
    lri = load_package()
    kind = case["kind"]
    Y = lri.SVDLikeRepresentation
    if kind == "solve":
        A, B, U, S, V = _solve_parts(case, seed)
        prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B), Y(U, S, V),
                                   (0.0, case["steps"] * case["dt"]))
        return dict(kind=kind, lri=lri, prob=prob, alg=lri.UnconventionalAlgorithm(lri.RK4(case["nsub"])),
                    dt=case["dt"], keep=case["keep"])
    if kind == "laplace":
        A, U, S, V, dt = _laplace_parts(case, seed)
        prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, A), Y(U, S, V), (0.0, case["steps"] * dt))
        return dict(kind=kind, lri=lri, prob=prob, alg=lri.UnconventionalAlgorithm(lri.RK4(case["nsub"])), dt=dt,
                    keep=False)
    if kind == "data":
        snaps, U, S, V = _data_parts(case, seed)
        return dict(kind=kind, lri=lri, prob=lri.MatrixDataProblem(snaps, Y(U, S, V)),
                    alg=lri.UnconventionalAlgorithm(), dt=None, keep=True)
    if kind in ("ensemble", "adaptive"):
        e = _members(case, seed)
        alg = _algorithm(lri, case)
        rcap = np.full(case["count"], case["rcap"]) if kind == "adaptive" else e["r"]
        b = lri.Batch(e["n"], e["m"], e["r"], alg, lri.SylvesterTridiagOperator.kind, case["precision"], r_cap=rcap)
        if case["precision"] != "fp64":
            b.apply_tuning()
        if kind == "adaptive":
            pad = case["rcap"] - case["r"]
            grow = torch.nn.functional.pad
            U0, V0, S0 = grow(e["U"], (0, pad)), grow(e["V"], (0, pad)), grow(e["S"], (0, pad, 0, pad))
            U0, V0, S0 = (x.transpose(1, 2).reshape(-1) for x in (U0, V0, S0))
        else:
            c = e["cols"]
            U0 = _packed(e["U"].transpose(1, 2), c[:, :, None] & e["rows"][:, None, :])
            V0 = _packed(e["V"].transpose(1, 2), c[:, :, None] & e["cols_m"][:, None, :])
            S0 = _packed(e["S"].transpose(1, 2), c[:, :, None] & c[:, None, :])
        three = torch.ones((1, 3, 1), dtype=torch.bool, device=DEV)
        b.opA[:int(3 * e["n"].sum())].copy_(_packed(e["A"], three & e["rows"][:, None, :]))
        b.opB[:int(3 * e["m"].sum())].copy_(_packed(e["B"], three & e["cols_m"][:, None, :]))
        U0, S0, V0 = (x.to(b.dtype) for x in (U0, S0, V0))
        state = dict(kind=kind, b=b, U0=U0, S0=S0, V0=V0, steps=case["steps"], count=case["count"])
        if kind == "adaptive":
            state.update(shape=(case["n"], case["m"], case["rcap"]))
        return state
    if kind == "mixed":
        e = _members(case, seed)
        hU, hS, hV, hA, hB = (e[k].cpu().numpy() for k in ("U", "S", "V", "A", "B"))
        r = e["r"]
        factors = [Y(hU[i, :, :r[i]].copy(), hS[i, :r[i], :r[i]].copy(), hV[i, :, :r[i]].copy())
                   for i in range(case["count"])]
        ops = [lri.SylvesterTridiagOperator(hA[i], hB[i]) for i in range(case["count"])]
        rcap = [int(r.max())] * case["count"]
        ens = lri.MixedEnsemble(factors, ops, lri.UnconventionalAlgorithm(lri.RK4(1)),
                                lri.SylvesterTridiagOperator.kind, r_cap=rcap)
        start = [(b.U.clone(), b.S.clone(), b.V.clone()) for _, _, b, _ in ens.parts]
        return dict(kind=kind, ens=ens, start=start, steps=case["steps"], shape=(case["n"], case["m"], int(r.max())))
    if kind == "stream":
        snaps, (U, s, V) = _snapshots(case, seed)
        eng = lri.DataStreamEngine(case["n"], case["m"], case["K"], case["rmax"], 1e-6, 1, "fp32")
        eng.bind(Y(U.cpu().numpy(), np.diag(s.cpu().numpy()), V.cpu().numpy()))
        return dict(kind=kind, eng=eng, snaps=snaps)
    if kind == "burgers":
        U, s, V, nu, h, dt = _burgers_parts(case, seed)
        op = lri.BurgersOperator(h, nu, alpha=0.0, beta=-0.5)
        eng = lri.BurgersLargeEngine(op, case["n"], case["m"], case["r"], case["r"], 1e-4, lri.RK4(case["nsub"]),
                                     case["r"], "fp32")
        eng.bind(Y(U, np.diag(s), V))
        return dict(kind=kind, eng=eng, dt=dt)
    A0, B, theta, U, S, V, P, D, Q = _gradient_parts(case, seed)
    prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A0, B, theta), Y(U, S, V), (0.0, case["steps"] * 1e-4))
    return dict(kind=kind, lri=lri, prob=prob, alg=lri.UnconventionalAlgorithm(lri.RK4(1)), target=Y(P, D, Q),
                every=case["every"])


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _field(b, n, m, rc, count):
    """Y = U S V^T of a batch whose members have one shape."""
    U, S, V = (x[:count * k].view(count, rc, -1) for x, k in ((b.U, n * rc), (b.S, rc * rc), (b.V, m * rc)))
    return torch.bmm(U.transpose(1, 2), torch.bmm(S.transpose(1, 2), V))


def run(state):
    kind = state["kind"]
    if kind in ("solve", "laplace", "data"):
        sol = state["lri"].solve(state["prob"], state["alg"], state["dt"], save_everystep=state["keep"])
        return [(Y.U, Y.S, Y.V) for Y in sol.Y[1:]]
    if kind in ("ensemble", "adaptive"):
        b = state["b"]
        k = state["U0"].numel(), state["S0"].numel(), state["V0"].numel()
        b.U[:k[0]].copy_(state["U0"])
        b.S[:k[1]].copy_(state["S0"])
        b.V[:k[2]].copy_(state["V0"])
        b.bind()
        for j in range(state["steps"]):
            b.step(j * ENSEMBLE_DT, ENSEMBLE_DT)
        if kind == "adaptive":
            n, m, rc = state["shape"]
            return {"Y": _field(b, n, m, rc, state["count"])}
        return {"U": b.U[:k[0]], "S": b.S[:k[1]], "V": b.V[:k[2]]}
    if kind == "mixed":
        ens = state["ens"]
        for (_, _, b, _), (U, S, V) in zip(ens.parts, state["start"]):
            b.U.copy_(U)
            b.S.copy_(S)
            b.V.copy_(V)
            b.bind()
        for j in range(state["steps"]):
            ens.step(j * ENSEMBLE_DT, ENSEMBLE_DT)
        n, m, rc = state["shape"]
        return {prec: _field(b, n, m, rc, b.count) for prec, _, b, _ in ens.parts}
    if kind == "stream":
        # forward through the snapshots and back to the first one
        eng, A = state["eng"], state["snaps"]
        path = list(range(len(A))) + list(range(len(A) - 2, -1, -1))
        for p, q in zip(path, path[1:]):
            eng.step(A[p], A[q])
        return {"Y": _large_field(eng)}
    if kind == "burgers":
        state["eng"].advance(state["dt"], 1)
        return {"Y": _large_field(state["eng"])}
    loss, theta, g = state["lri"].bug_gradient(state["prob"], state["alg"], 1e-4, state["target"], state["every"])
    return {"loss": loss, "theta": theta, "U": g.U, "S": g.S, "V": g.V}


def _large_field(eng):
    U, S, V = eng.U.view(eng.R, eng.n), eng.S.view(eng.R, eng.R), eng.V.view(eng.R, eng.m)
    return U.T @ (S.T @ V)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _step_work(n, m, r, nsub, esize, alg="bug"):
    """Factors and operators read, factors written; the flops of one step (arrays: per member)."""
    nm = np.asarray(n, np.float64) + m
    r = np.asarray(r, np.float64)
    by = (2 * nm * r + 2 * r * r + 3 * nm) * esize
    if alg == "ra":
        fl = (2 + 8 * nsub + 16 + 8 + 8) * nm * r * r + (20 * nsub + 30) * nm * r + (64 * nsub + 160) * r**3
    else:
        fl = (12 + 8 * nsub) * nm * r * r + (36 * nsub + 5) * nm * r + (4 + 16 * nsub) * r**3
        if alg == "ksl":
            fl = 2 * fl
    return by, fl


def work(case):
    kind = case["kind"]
    if kind in ("solve", "laplace"):
        n, m = case["n"], case.get("m", case["n"])
        by, fl = _step_work(n, m, case["r"], case["nsub"], 8)
        return {"bytes": float(by), "flops": float(fl * case["steps"])}
    if kind == "data":
        N, r, k = case["n"], case["r"], case["steps"]
        return {"bytes": 8.0 * N * N * (k + 1) + 8.0 * k * (2 * N * r + r * r),
                "flops": k * (6.0 * N * N * r + 16.0 * N * r * r)}
    if kind in ("ensemble", "mixed", "adaptive"):
        cnt = case["count"]
        if kind == "ensemble":
            n = m = (case["nmin"] + case["nmax"]) / 2
        else:
            n, m = case["n"], case["m"]
        r = np.full(1, case["r"]) if kind == "adaptive" else np.arange(case["rmin"], case["rmax"] + 1)
        by, fl = _step_work(n, m, r, 1, 4 if case.get("precision", "fp32") == "fp32" else 8,
                            "ra" if kind == "adaptive" else case.get("alg", "bug"))
        out = {"bytes": cnt * float(np.mean(by)), "flops": cnt * case["steps"] * float(np.mean(fl))}
        if kind != "ensemble":
            out["bytes"] += 4.0 * cnt * n * m
            out["flops"] += 2.0 * cnt * n * m * float(np.mean(r))
        return out
    if kind == "stream":
        n, m, K, s = case["n"], case["m"], case["K"], case["snaps"]
        k = 2 * (s - 1)
        return {"bytes": 4.0 * n * m * (s + 1) + 8.0 * K * (n + m),
                "flops": k * (6.0 * n * m * K + 40.0 * (n + m) * K * K) + 2.0 * n * m * K}
    if kind == "burgers":
        n, m, r = case["n"], case["m"], case["r"]
        pairs = lambda k: k * (k + 1) / 2  # noqa: E731
        stage = (n + m) * r * r + (n + m) * pairs(r) * r + 2 * n * (2 * r) ** 2 + 2 * (2 * r) ** 3 + n * pairs(2 * r) * 2 * r
        tens = (n + m) * pairs(r) * r + m * pairs(2 * r) * 2 * r
        return {"bytes": 4.0 * (2 * (n + m) * r + m) + 4.0 * n * m,
                "flops": 2.0 * (4 * case["nsub"] * stage + tens) + 2.0 * n * m * r}
    by, fl = _step_work(case["n"], case["m"], case["r"], 1, 8)
    return {"bytes": 2.0 * float(by), "flops": 5.0 * case["steps"] * float(fl)}


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch
# ---------------------------------------------------------------------------

def _tri_mul(T, X):
    """Tridiagonal operators [sub, dia, sup] (..., 3, N) times panels (..., N, r), zero outside."""
    sub, dia, sup = T[..., 0, :, None], T[..., 1, :, None], T[..., 2, :, None]
    Z = torch.zeros_like(X[..., :1, :])
    down = torch.cat([Z, X[..., :-1, :]], dim=-2)
    up = torch.cat([X[..., 1:, :], Z], dim=-2)
    return sub * down + dia * X + sup * up


def _rk4(f, y, dt, nsub):
    h = dt / nsub
    for _ in range(nsub):
        k1 = f(y)
        k2 = f(y + 0.5 * h * k1)
        k3 = f(y + 0.5 * h * k2)
        k4 = f(y + h * k3)
        y = y + h * (k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6)
    return y


def _qr(K, cols=None, positive=False):
    """Thin QR of (padded) panels with Householder's signs (or a positive diagonal of R); (Q, R)."""
    Q, R = torch.linalg.qr(K)
    d = torch.where(torch.diagonal(R, dim1=-2, dim2=-1) < 0, -1.0, 1.0).to(F64)
    Q, R = Q * d[..., None, :], R * d[..., :, None]
    if not positive:
        # the reflections' signs: R_jj = -sign(pivot), from the elimination of Q's top block
        r = Q.shape[-1]
        T = Q[..., :r, :].clone()
        s = torch.ones_like(d)
        for j in range(r):
            s[..., j] = torch.where(T[..., j, j] < 0, 1.0, -1.0)
            piv = T[..., j, j] - s[..., j]
            col = T[..., j + 1:, j] / piv[..., None]
            T[..., j + 1:, j + 1:] -= col[..., :, None] * T[..., j, j + 1:][..., None, :]
        Q, R = Q * s[..., None, :], R * s[..., :, None]
    if cols is not None:
        Q = Q * cols[..., None, :]
        R = R * cols[..., :, None]
    return Q, R


def _t(X):
    return X.transpose(-1, -2)


def _k_flow(A, V, B):
    G, P = _t(V) @ V, _t(V) @ _tri_mul(B, V)
    return lambda K: _tri_mul(A, K) @ G + K @ _t(P)


def _s_flow(U, V, A, B, sign=1.0):
    PU, GU, PV, GV = _t(U) @ _tri_mul(A, U), _t(U) @ U, _t(V) @ _tri_mul(B, V), _t(V) @ V
    return lambda S: sign * (PU @ S @ GV + GU @ S @ _t(PV))


def _bug(U, S, V, A, B, dt, nsub, cols=None, positive=False):
    U1 = _qr(_rk4(_k_flow(A, V, B), U @ S, dt, nsub), cols, positive)[0]
    V1 = _qr(_rk4(_k_flow(B, U, A), V @ _t(S), dt, nsub), cols, positive)[0]
    S0 = (_t(U1) @ U) @ S @ _t(_t(V1) @ V)
    return U1, _rk4(_s_flow(U1, V1, A, B), S0, dt, nsub), V1


def _ksl(U, S, V, A, B, dt, cols, positive, primal):
    if primal:
        U, S = _qr(_rk4(_k_flow(A, V, B), U @ S, dt, 1), cols, positive)
        S = _rk4(_s_flow(U, V, A, B, -1.0), S, dt, 1)
        V, R = _qr(_rk4(_k_flow(B, U, A), V @ _t(S), dt, 1), cols, positive)
        return U, _t(R), V
    V, R = _qr(_rk4(_k_flow(B, U, A), V @ _t(S), dt, 1), cols, positive)
    S = _rk4(_s_flow(U, V, A, B, -1.0), _t(R), dt, 1)
    U, S = _qr(_rk4(_k_flow(A, V, B), U @ S, dt, 1), cols, positive)
    return U, S, V


def _truncate(P, s, Qt, tol, rmin, rmax):
    tail, r = 0.0, len(s)
    while tail < tol * tol and r > 0:
        tail += float(s[r - 1]) ** 2
        r -= 1
    r = min(max(min(r + 1, rmax), rmin), len(s))
    return P[:, :r], s[:r], Qt[:r]


def _adaptive_y(U, S, V, A, B, dt, steps, tol, rcap):
    """Rank-adaptive steps of one member; its Y."""
    for _ in range(steps):
        K1 = _rk4(_k_flow(A, V, B), U @ S, dt, 1)
        L1 = _rk4(_k_flow(B, U, A), V @ S.T, dt, 1)
        Uh, Vh = torch.linalg.qr(torch.cat([K1, U], 1))[0], torch.linalg.qr(torch.cat([L1, V], 1))[0]
        S1 = _rk4(_s_flow(Uh, Vh, A, B), (Uh.T @ U) @ S @ (Vh.T @ V).T, dt, 1)
        P, s, Qt = _truncate(*torch.linalg.svd(S1), tol, 1, rcap)
        U, S, V = Uh @ P, torch.diag(s), Vh @ Qt.T
    return U @ S @ V.T


def _host(x):
    return torch.from_numpy(np.ascontiguousarray(x))


def _exact_solve(A, B, U, S, V, dt, nsub, steps, keep):
    A, B = (torch.stack([_host(x) for x in T]) for T in (A, B))
    U, S, V = _host(U), _host(S), _host(V)
    out = []
    for _ in range(steps):
        U, S, V = _bug(U, S, V, A, B, dt, nsub)
        out.append((U, S, V))
    return out if keep else out[-1:]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, B, U, S, V = _solve_parts(case, seed)
        return _exact_solve(A, B, U, S, V, case["dt"], case["nsub"], case["steps"], case["keep"])
    if kind == "laplace":
        A, U, S, V, dt = _laplace_parts(case, seed)
        return _exact_solve(A, A, U, S, V, dt, case["nsub"], case["steps"], False)
    if kind == "data":
        snaps, U, S, V = _data_parts(case, seed)
        snaps, U, S, V = [_host(x) for x in snaps], _host(U), _host(S), _host(V)
        out = []
        for prev, cur in zip(snaps, snaps[1:]):
            D = cur - prev
            U1, V1 = _qr(U @ S + D @ V)[0], _qr(V @ S.T + D.T @ U)[0]
            S = (U1.T @ U) @ S @ (V1.T @ V).T + U1.T @ D @ V1
            U, V = U1, V1
            out.append((U, S, V))
        return out
    if kind in ("ensemble", "mixed"):
        e = _members(case, seed)
        U, S, V, A, B, cols = (e[k] for k in ("U", "S", "V", "A", "B", "cols"))
        pos = case.get("precision") == "df"
        c = cols.to(F64)
        for _ in range(case["steps"]):
            if case.get("alg") == "ksl":
                U, S, V = _ksl(U, S, V, A, B, 0.5 * ENSEMBLE_DT, c, pos, True)
                U, S, V = _ksl(U, S, V, A, B, 0.5 * ENSEMBLE_DT, c, pos, False)
            else:
                U, S, V = _bug(U, S, V, A, B, ENSEMBLE_DT, 1, c, pos)
        if kind == "mixed":
            # members with cores beyond the FP32 class's conditioning are advanced in double-float
            hard = torch.from_numpy(2.0 ** (e["r"] - 1) > mixed_limit()).to(DEV)
            out = {}
            for prec, sel in (("fp32", ~hard), ("df", hard)):
                if bool(sel.any()):
                    out[prec] = torch.bmm(U[sel], torch.bmm(S[sel], _t(V[sel])))
            return out
        return {"U": _packed(_t(U), cols[:, :, None] & e["rows"][:, None, :]),
                "S": _packed(_t(S), cols[:, :, None] & cols[:, None, :]),
                "V": _packed(_t(V), cols[:, :, None] & e["cols_m"][:, None, :])}
    if kind == "adaptive":
        e = {k: v.cpu() if torch.is_tensor(v) else v for k, v in _members(case, seed).items()}
        return {"Y": torch.stack([_adaptive_y(e["U"][i], e["S"][i], e["V"][i], e["A"][i], e["B"][i], ENSEMBLE_DT,
                                              case["steps"], 1e-6, case["rcap"]) for i in range(case["count"])])}
    if kind == "stream":
        snaps, (U, s, V) = _snapshots(case, seed)
        U, S, V = U.float().double(), torch.diag(s.float().double()), V.float().double()
        path = list(range(len(snaps))) + list(range(len(snaps) - 2, -1, -1))
        for p, q in zip(path, path[1:]):
            D = (snaps[q].double() - snaps[p].double()).T
            Uh = torch.linalg.qr(torch.cat([U @ S + D @ V, U], 1))[0]
            Vh = torch.linalg.qr(torch.cat([V @ S.T + D.T @ U, V], 1))[0]
            S1 = (Uh.T @ U) @ S @ (Vh.T @ V).T + Uh.T @ (D @ Vh)
            P, s, Qt = _truncate(*torch.linalg.svd(S1), 1e-6, 1, case["rmax"])
            U, S, V = Uh @ P, torch.diag(s), Vh @ Qt.T
        return {"Y": U @ S @ V.T}
    if kind == "burgers":
        return {"Y": _exact_burgers(case, seed)}
    return _exact_gradient(case, seed)


def mixed_limit():
    """Core conditioning up to which the mixed ensemble keeps a member in FP32 (its documented default)."""
    return 2.0 ** 21


def _exact_burgers(case, seed):
    """One rank-adaptive step: F(Y) = (Dxx Y) diag(nu) - Dx(Y*Y)/2 on factors, products by 3-tensors."""
    Uh_, s, Vh_, nu, h, dt = _burgers_parts(case, seed)
    U, V, nu = (torch.from_numpy(x).to(DEV) for x in (Uh_, Vh_, nu))
    S = torch.diag(torch.from_numpy(s).to(DEV))
    nsub, r = case["nsub"], case["r"]
    dxx = lambda X: (torch.roll(X, -1, 0) - 2 * X + torch.roll(X, 1, 0)) / h**2  # noqa: E731
    dx = lambda X: (torch.roll(X, -1, 0) - torch.roll(X, 1, 0)) / (2 * h)  # noqa: E731

    def rows(f, X, step=2048):
        return torch.cat([f(X[i:i + step]) for i in range(0, X.shape[0], step)])

    def tensor(X, W):
        """sum_j X_ja X_jb W_jc as an (a b) x c matrix."""
        k = X.shape[1]
        out = torch.zeros((k * k, W.shape[1]), device=DEV, dtype=F64)
        for i in range(0, X.shape[0], 1024):
            x = X[i:i + 1024]
            out += (x[:, :, None] * x[:, None, :]).reshape(x.shape[0], -1).T @ W[i:i + 1024]
        return out

    def square(X, T):
        """rows sum_ab X_ia X_ib T_abc"""
        return rows(lambda x: (x[:, :, None] * x[:, None, :]).reshape(x.shape[0], -1) @ T, X)

    TV, Nv = tensor(V, V), V.T @ (nu[:, None] * V)
    K1 = _rk4(lambda K: dxx(K) @ Nv - 0.5 * dx(square(K, TV)), U @ S, dt, nsub)
    # F(U L^T)^T U = nu L (U^T Dxx U)^T + (1/2) sum_ab L_ja L_jb (sum_i U_ia U_ib (Dx U)_ic)
    TU, Uxx = tensor(U, dx(U)), U.T @ dxx(U)
    L1 = _rk4(lambda L: nu[:, None] * (L @ Uxx.T) + 0.5 * square(L, TU), V @ S.T, dt, nsub)
    Uh, Vh = torch.linalg.qr(torch.cat([K1, U], 1))[0], torch.linalg.qr(torch.cat([L1, V], 1))[0]
    TV, Nv, Axx = tensor(Vh, Vh), Vh.T @ (nu[:, None] * Vh), Uh.T @ dxx(Uh)
    S1 = _rk4(lambda Z: Axx @ Z @ Nv - 0.5 * Uh.T @ dx(square(Uh @ Z, TV)), (Uh.T @ U) @ S @ (Vh.T @ V).T, dt, nsub)
    P, s, Qt = _truncate(*torch.linalg.svd(S1), 1e-4, r, r)
    return (Uh @ P * s) @ (Vh @ Qt.T).T


def _exact_gradient(case, seed):
    A0, B, theta, U, S, V, P, D, Q = _gradient_parts(case, seed)
    T0, B = (torch.stack([_host(x) for x in T]) for T in (A0, B))
    th, U0, S0, V0 = (_host(x).requires_grad_() for x in (theta, U, S, V))
    zero = torch.zeros_like(th)
    A = T0 + torch.stack([zero, th, zero])
    u, s, v = U0, S0, V0
    for _ in range(case["steps"]):
        # (the signs of the bases' columns cancel in the loss and its gradient)
        u1 = torch.linalg.qr(_rk4(_k_flow(A, v, B), u @ s, 1e-4, 1))[0]
        v1 = torch.linalg.qr(_rk4(_k_flow(B, u, A), v @ s.T, 1e-4, 1))[0]
        s = _rk4(_s_flow(u1, v1, A, B), (u1.T @ u) @ s @ (v1.T @ v).T, 1e-4, 1)
        u, v = u1, v1
    W, Qt = _host(P) @ _host(D), _host(Q)
    loss = (torch.trace(s.T @ (u.T @ u) @ s @ (v.T @ v)) - 2 * torch.trace(s.T @ (u.T @ W) @ (Qt.T @ v))
            + torch.sum((W.T @ W) * (Qt.T @ Qt)))
    loss.backward()
    return {"loss": float(loss.detach()), "theta": th.grad, "U": U0.grad, "S": S0.grad, "V": V0.grad}
