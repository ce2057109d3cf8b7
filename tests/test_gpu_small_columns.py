"""Bases from panels whose columns are so small that their squares leave the
type's exponent range: orthonormal, and the ones of the same panel scaled by a
power of two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def instance(seed, n, m, r):
    g = np.random.default_rng(seed)
    A = (g.uniform(0.5, 1, n), -2 - g.uniform(0, 1, n), g.uniform(0.5, 1, n))
    B = (g.uniform(0.5, 1, m), -2 - g.uniform(0, 1, m), g.uniform(0.5, 1, m))
    U, V = (np.linalg.qr(g.standard_normal((k, r)))[0] for k in (n, m))
    return A, B, U, np.diag(2.0 ** (-np.arange(1, r + 1) / 4.0)), V


# The flow is linear: a core scaled by a power of two gives the same bases and
# the scaled core, to the rounding of two FP64 steps at condition 2^(r/4).
@pytest.mark.parametrize("kind", ["bug", "ksl"])
@pytest.mark.parametrize("n,m,r", [(40, 36, 4), (300, 257, 16), (64, 70, 33)])
@pytest.mark.parametrize("power", [-518, -525, -532, -560])
def test_fp64_steps_scale(lri, kind, n, m, r, power):
    A, B, U, S, V = instance(n + r, n, m, r)
    alg = {"bug": lri.UnconventionalAlgorithm(lri.RK4(1)),
           "ksl": lri.ProjectorSplitting(lri.PrimalLieTrotter(), lri.RK4(1))}[kind]

    def run(scale):
        prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B),
                                   lri.SVDLikeRepresentation(U, S * scale, V), (0.0, 2e-2))
        return lri.solve(prob, alg, 1e-2).Y[-1]

    scale = 2.0 ** power
    y, ref = run(scale), run(1.0)
    for X in (y.U, y.V):
        assert np.abs(X.T @ X - np.eye(r)).max() <= 1e-13
    for a, b in ((y.U, ref.U), (y.S / scale, ref.S), (y.V, ref.V)):
        assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("n,m", [(50, 40), (700, 33)])
def test_fp64_graded_columns(lri, n, m):
    """Columns from 1 down to 2^-560 beside each other (the panels are U S)."""
    _, _, U, _, V = instance(9, n, m, 9)
    S = np.diag(2.0 ** np.array([0, -100, -300, -450, -512, -520, -528, -540, -560.0]))
    prob = lri.MatrixDEProblem(lri.ZeroOperator(), lri.SVDLikeRepresentation(U, S, V), (0.0, 1.0))
    for alg in (lri.UnconventionalAlgorithm(lri.RK4(1)), lri.ProjectorSplitting(lri.PrimalLieTrotter(), lri.RK4(1))):
        y = lri.solve(prob, alg, 1.0).Y[-1]
        for X, X0 in ((y.U, U), (y.V, V)):
            assert np.abs(X.T @ X - np.eye(9)).max() <= 1e-14 * 9
            # every column along the one it came from
            assert np.abs(np.abs(np.sum(X * X0, axis=0)) - 1).max() <= 1e-12


# Rank-adaptive: the old basis's columns repeat the new panel's, and what is
# left of them after the elimination is rounding of the small rows.
@pytest.mark.parametrize("precision,small,tol", [("fp32", 1e-13, 1e-5), ("fp32", 3e-14, 1e-5), ("fp32", 3e-15, 1e-5),
                                                 ("df", 1e-6, 1e-11), ("df", 1e-7, 1e-11), ("df", 1e-8, 1e-11)])
def test_rank_adaptive_small_remainders(lri, precision, small, tol):
    n, m, r = 90, 70, 4
    g = np.random.default_rng(3)
    U, V = (np.vstack([np.eye(r), small * g.standard_normal((k - r, r))]) for k in (n, m))
    S = np.diag([0.7, 0.3, 0.19, 0.11])
    alg = lri.RankAdaptiveUnconventionalAlgorithm(1e-9, rmax=2 * r, K_alg=lri.RK4(1), rmin=2 * r)
    prob = lri.MatrixDEProblem(lri.ZeroOperator(), lri.SVDLikeRepresentation(U, S, V), (0.0, 1.0))
    y = lri.solve(prob, alg, 1.0, precision=precision).Y[-1]
    assert y.S.shape == (2 * r, 2 * r)
    for X in (y.U, y.V):
        assert np.abs(X.T @ X - np.eye(2 * r)).max() <= tol


# Bases that are orthonormal to a few 1e-12 only: their Gram matrices' last bits
# count, also where the panels' entries lie below the FP32 range.
def nearly_orthonormal(g, X):
    return X @ (np.eye(X.shape[1]) + 1.5e-12 * g.standard_normal((X.shape[1], X.shape[1])))


@pytest.mark.parametrize("n,m,r", [(40, 36, 4), (300, 257, 16), (70, 300, 33)])
@pytest.mark.parametrize("power", [-90, -150, -300])
def test_gram_terms_of_small_panels(lri, n, m, r, power):
    A, B, U, S, V = instance(n + r, n, m, r)
    g = np.random.default_rng(1)
    U, V = nearly_orthonormal(g, U), nearly_orthonormal(g, V)

    def run(scale):
        prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B),
                                   lri.SVDLikeRepresentation(U, S * scale, V), (0.0, 0.1))
        return lri.solve(prob, lri.UnconventionalAlgorithm(lri.RK4(1)), 0.1).Y[-1]

    scale = 2.0 ** power
    y, ref = run(scale), run(1.0)
    # FP64 rounding at condition 2^(r/4) <= 2^8; without E the bases move by 1e-13 and more
    for a, b in ((y.U, ref.U), (y.S / scale, ref.S), (y.V, ref.V)):
        assert np.linalg.norm(a - b) <= 2e-14 * 2 ** (r / 8) * np.linalg.norm(b)


@pytest.mark.parametrize("n,m,r", [(40, 36, 4), (300, 257, 16)])
@pytest.mark.parametrize("power", [-90, -150])
def test_gradients_of_small_panels(lri, n, m, r, power):
    A, B, U, S, V = instance(n + r, n, m, r)
    g = np.random.default_rng(1)
    U, V = nearly_orthonormal(g, U), nearly_orthonormal(g, V)
    P, Q = (np.linalg.qr(g.standard_normal((k, 5)))[0] for k in (n, m))
    D = np.diag(2.0 ** -np.arange(5.0))

    def run(scale):
        prob = lri.MatrixDEProblem(lri.SylvesterTridiagOperator(A, B),
                                   lri.SVDLikeRepresentation(U, S * scale, V), (0.0, 0.1))
        _, theta, b = lri.bug_gradient(prob, lri.UnconventionalAlgorithm(lri.RK4(1)), 0.1,
                                       lri.SVDLikeRepresentation(P, D * scale, Q))
        return theta / scale ** 2, b.U / scale ** 2, b.S / scale, b.V / scale ** 2

    for a, b in zip(run(2.0 ** power), run(1.0)):
        assert np.linalg.norm(a - b) <= 2e-13 * 2 ** (r / 8) * np.linalg.norm(b)
