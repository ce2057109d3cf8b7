"""FP64 BUG steps of small batches on thread-block clusters (the rows of each
side split over a cluster, the core's columns over another) against the
oracle: factors, not only Y (both use Householder's signs), at row counts
with remainders, empty CTAs and fewer rows than columns per CTA, one-column
to 64-column cores, batches of uneven members, data streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# FP64 factors of cores with condition number 2^(r/4) <= 2^16 over three
# steps: rounding grows to about 1e-16 * 2^16 * sqrt(n r) < 1e-9
TOL = 1e-9


def instance(seed, n, m, r):
    g = np.random.default_rng(seed)
    A = (g.uniform(0.5, 1, n), -2 - g.uniform(0, 1, n), g.uniform(0.5, 1, n))
    B = (g.uniform(0.5, 1, m), -2 - g.uniform(0, 1, m), g.uniform(0.5, 1, m))
    U, V = (np.linalg.qr(g.standard_normal((k, r)))[0] for k in (n, m))
    return A, B, U, np.diag(2.0 ** (-np.arange(1, r + 1) / 4.0)), V


def close(a, b):
    return np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)


@pytest.mark.parametrize("scheme,nsub", [("RK4", 2), ("Heun", 1), ("Euler", 3)])
@pytest.mark.parametrize("shapes", [[(8, 9, 1)], [(33, 17, 5)], [(17, 130, 16)], [(300, 257, 32)], [(64, 70, 64)],
                                    [(100, 64, 33)], [(512, 40, 7), (31, 300, 20), (64, 64, 3)],
                                    [(40 + 3 * i, 60 - i, 2 + i % 5) for i in range(21)]])
def test_wide_step_matches_oracle(lri, oracle, shapes, scheme, nsub):
    dt, k = 1e-2, 3
    ins = [instance(10 + i, *s) for i, s in enumerate(shapes)]
    probs = [lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B), lri.SVDLikeRepresentation(U, S, V), (0.0, k * dt))
             for A, B, U, S, V in ins]
    got = lri.solve_ensemble(probs, lri.UnconventionalAlgorithm(getattr(lri, scheme)(nsub)), dt, precision="fp64")
    for (A, B, U, S, V), y in zip(ins, got):
        po = oracle.MatrixDEProblem(oracle.SylvesterTridiagOp(A, B), oracle.SVDLikeRepresentation(U, S, V), (0.0, k * dt))
        yo = oracle.solve(po, oracle.UnconventionalAlgorithm(getattr(oracle, scheme)(nsub)), dt).Y[-1]
        assert close(y.U, yo.U) and close(y.S, yo.S) and close(y.V, yo.V)


def test_wide_step_full_gram_form(lri, oracle):
    """A basis that is not orthonormal to 2^-36 takes the full Gram product."""
    A, B, U, S, V = instance(3, 120, 90, 6)
    U = U * (1 + 1e-6 * np.arange(6))
    V = V @ (np.eye(6) + 1e-4 * np.ones((6, 6)))
    po = oracle.MatrixDEProblem(oracle.SylvesterTridiagOp(A, B), oracle.SVDLikeRepresentation(U, S, V), (0.0, 0.02))
    pg = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B), lri.SVDLikeRepresentation(U, S, V), (0.0, 0.02))
    y = lri.solve(pg, lri.UnconventionalAlgorithm(lri.RK4(2)), 0.01).Y[-1]
    yo = oracle.solve(po, oracle.UnconventionalAlgorithm(oracle.RK4(2)), 0.01).Y[-1]
    assert close(y.U, yo.U) and close(y.S, yo.S) and close(y.V, yo.V)


@pytest.mark.parametrize("n,m,r", [(100, 100, 12), (8, 70, 3), (131, 33, 32), (200, 210, 64)])
def test_wide_data_step_matches_oracle(lri, oracle, n, m, r):
    g = np.random.default_rng(n)
    _, _, U, S, V = instance(n, n, m, r)
    snaps = [U @ S @ V.T]
    for _ in range(3):
        snaps.append(snaps[-1] + 0.05 * g.standard_normal((n, m)))
    sg = lri.solve(lri.MatrixDataProblem(snaps, lri.SVDLikeRepresentation(U, S, V)), lri.UnconventionalAlgorithm())
    so = oracle.solve(oracle.MatrixDataProblem(snaps, oracle.SVDLikeRepresentation(U, S, V)),
                      oracle.UnconventionalAlgorithm())
    for y, yo in zip(sg.Y, so.Y):
        assert close(y.U, yo.U) and close(y.S, yo.S) and close(y.V, yo.V)


def test_wide_graph_and_single_steps_agree(lri):
    """One five-step call (a captured graph) and five calls give the same bits,
    also after binding new factors."""
    A, B, U, S, V = instance(5, 210, 190, 9)
    b = lri.Batch([210], [190], [9], lri.UnconventionalAlgorithm(lri.RK4(1)), lri.SylvesterTridiagOperator.kind, "fp64")
    out = []
    for multi in (True, False):
        b.upload([lri.SVDLikeRepresentation(U, S, V)], [lri.SylvesterTridiagOperator(A, B)])
        if multi:
            b.step(0.0, 0.01, 5)
        else:
            for j in range(5):
                b.step(0.01 * j, 0.01)
        b.check_status()
        out.append(b.download()[0])
    assert np.array_equal(out[0].U, out[1].U) and np.array_equal(out[0].S, out[1].S) and np.array_equal(out[0].V, out[1].V)


@pytest.mark.parametrize("n,m,r,scheme,nsub,steps", [(24, 20, 3, "RK4", 1, 3), (65, 40, 5, "Heun", 3, 2),
                                                      (17, 130, 9, "Euler", 2, 3), (257, 130, 32, "RK4", 2, 2),
                                                      (70, 64, 48, "RK4", 1, 1)])
def test_wide_gradient_matches_cpu_adjoint(lri, oracle, n, m, r, scheme, nsub, steps):
    """Loss gradient through the clusters' reverse steps against the NumPy
    adjoint: theta and all three input factors."""
    from oracle import lri_adjoint as AD
    g = np.random.default_rng(n + m)
    dt = 0.02
    A0 = (np.ones(n), -2.0 * np.ones(n), np.ones(n))
    B = (g.uniform(0.5, 1, m), -2.0 - g.uniform(0, 1, m), g.uniform(0.5, 1, m))
    theta = g.normal(0.0, 0.1, n)
    _, _, U, S, V = instance(n, n, m, r)
    S = S + 0.01 * g.standard_normal((r, r))
    P, Q = (np.linalg.qr(g.standard_normal((k, 6)))[0] for k in (n, m))
    d = 2.0 ** (-np.arange(1, 7) / 4.0)
    k = lri.n_steps((0.0, steps * dt), dt)
    _, tc, uc, sc, vc = AD.loss_and_grad(U, S, V, A0, theta, B, getattr(oracle, scheme)(nsub), dt, k, (P, d, Q),
                                         checkpoint_every=2)
    prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A0, B, theta), lri.SVDLikeRepresentation(U, S, V),
                               (0.0, steps * dt))
    _, tg, gr = lri.bug_gradient(prob, lri.UnconventionalAlgorithm(getattr(lri, scheme)(nsub)), dt,
                                 lri.SVDLikeRepresentation(P, np.diag(d), Q), checkpoint_every=2)
    for a, b in ((tg, tc), (gr.U, uc), (gr.S, sc), (gr.V, vc)):
        assert close(a, b)


# double-float steps by sides: clusters of every size, remainders and empty
# CTAs, scratch inside and outside the free panels, cores up to 64 columns;
# graded cores (kappa 2^(r-1)) take the shifted three-pass QR, a core with a
# zero singular value the Householder fallback
@pytest.mark.parametrize("grade", ["mild", "graded", "singular"])
@pytest.mark.parametrize("shapes", [[(9, 8, 1)], [(70, 33, 5)], [(64, 64, 64)], [(1000, 130, 33)], [(600, 517, 12)],
                                    [(64 + 7 * i, 300 - 5 * i, 3 + i % 9) for i in range(24)]])
def test_df_sides_match_oracle(lri, oracle, shapes, grade):
    dt, k = 1e-2, 3
    probs, refs = [], []
    for i, s in enumerate(shapes):
        A, B, U, S, V = instance(50 + i, *s)
        r = s[2]
        if grade == "graded":
            S = np.diag(2.0 ** -np.minimum(np.arange(1, r + 1), 31))
        if grade == "singular" and r > 1:
            S[-1, -1] = 0.0
        probs.append(lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B), lri.SVDLikeRepresentation(U, S, V), (0.0, k * dt)))
        refs.append(oracle.solve(oracle.MatrixDEProblem(oracle.SylvesterTridiagOp(A, B), oracle.SVDLikeRepresentation(U, S, V),
                                                        (0.0, k * dt)), oracle.UnconventionalAlgorithm(oracle.RK4(1)), dt).Y[-1])
    got = lri.solve_ensemble(probs, lri.UnconventionalAlgorithm(lri.RK4(1)), dt, precision="df")
    for y, yo in zip(got, refs):
        # 48-bit significands: rounding of Y about 1e-14 sqrt(n r) per step
        assert oracle.rel_fro_err(y.full(), yo.full()) <= 1e-11
        for X in (y.U, y.V):
            assert np.abs(X.T @ X - np.eye(X.shape[1])).max() <= 1e-11


# the step kernel keeps batches that fill the GPU with tall panels of high rank;
# both routes take the same factors (one step of the first instances agrees)
@pytest.mark.parametrize("count,n,r,sides", [(3, 768, 28, True), (480, 768, 28, False), (480, 128, 12, True)])
def test_df_route_by_cost(lri, count, n, r, sides):
    g = np.random.default_rng(3)
    U, V = (np.linalg.qr(g.standard_normal((n, r)))[0] for _ in range(2))
    Y = lri.SVDLikeRepresentation(U, np.diag(2.0 ** -np.arange(1, r + 1)), V)
    T = (g.uniform(0.5, 1, n), -2 - g.uniform(0, 1, n), g.uniform(0.5, 1, n))
    op = lri.SylvesterTridiagOperator(T, T)
    alg = lri.UnconventionalAlgorithm(lri.RK4(1))
    kind = lri._native.LRI_OP_SYLVESTER_TRIDIAG
    one = lri.Batch([n], [n], [r], alg, kind, "df")
    b = lri.Batch([n] * count, [n] * count, [r] * count, alg, kind, "df")
    assert (b.launches_per_step() > 4) == sides and one.launches_per_step() > 4
    for x, k in ((one, 1), (b, count)):
        x.upload([Y] * k, [op] * k)
        x.step(0.0, 1e-2)
        x.check_status()
    ref, got = one.download()[0].full(), b.download()[count - 1].full()
    one.close()
    b.close()
    # double-float: 48 bits through some hundred dependent operations per entry
    assert np.linalg.norm(got - ref) <= 1e-11 * np.linalg.norm(ref)
