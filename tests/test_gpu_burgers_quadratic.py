"""The quadratic terms of the large Burgers engine's K, L and S flows against
the oracle, on problems whose increment is mostly theirs: errors relative to
Q = Y - (the same step without the quadratic terms).

Y of amplitude 1 on modes with at least 10 grid points a period (4 on the
short grids), singular values 1 to 0.7, and a dt with |Q| about 0.2 |Y|, so that the kept and the dropped
singular values stay apart (0.6 and 0.2) and the truncated Y is as well
conditioned as the flows.  FP32 roundings of Y are 2^-24 |Y| = 3e-7 |Q| each, some ten
in a row 3e-6 |Q|.  Single-pass TF32 products in place of the split ones move Y
by 9e-5 to 3e-4 (S flow), 5e-5 to 2e-4 (L flow) and 3e-5 to 9e-5 |Q| (K flow),
a slice off by 1 % by more; the tolerance of 1e-5 |Q| shows each of them.

The part of the error along Q: roundings to nearest leave 1e-8 of it, but the
tensor cores' accumulators cut the bits below their last one at every
addition, half a unit of a sum that is half complete on average.  The S
flow's three products make at most 16 such additions at the sums' size (4, 8
and 4): 16 * 2^-25 = 5e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(n, m, r, alpha, beta, seed=4):
    g = np.random.default_rng(seed)
    k = max(1, n // (5 * r)) * np.arange(1, (r + 1) // 2 + 1)  # multiples: their products fall on the modes again
    x = 2 * np.pi * np.outer(np.arange(n), k) / n
    F = np.hstack([np.sin(x), np.cos(x)])[:, :r]
    U = np.linalg.qr(F @ np.linalg.qr(g.standard_normal((r, r)))[0])[0]
    V = np.linalg.qr(g.standard_normal((m, r)))[0]
    S = np.diag(np.linspace(1.0, 0.7, r)) * np.sqrt(n * m / r)
    Y = U @ S @ V.T
    dx = lambda X: (np.roll(X, -1, 0) - np.roll(X, 1, 0)) / 2  # grid spacing 1
    dt = 0.25 * np.linalg.norm(Y) / np.linalg.norm(alpha * dx(Y) * Y + beta * dx(Y * Y))
    return U, S, V, g.uniform(0.01, 0.05, m), dt


# (n, m, r, substeps, alpha, beta): the flow kernels' two widths, the S flow's
# tensor-core form (two to four chunks), the panels' form with tiles shared by
# four, two and no CTAs, one and several launches of the K flow
CASES = [(97, 130, 16, 8, -1.0, 0.0), (129, 65, 17, 9, 0.0, -0.5), (100, 191, 32, 8, -0.5, -0.25),
         (160, 150, 33, 8, -1.0, 0.0), (131, 140, 49, 8, 0.0, -0.5), (140, 129, 64, 8, -0.4, -0.3),
         (300, 290, 57, 11, -0.2, -0.4), (6001, 131, 41, 8, -0.4, -0.3), (400, 6001, 49, 8, 0.0, -0.5),
         (9999, 400, 64, 8, -0.4, -0.3), (260, 9999, 35, 8, -0.5, -0.2)]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 1e-5)])
@pytest.mark.parametrize("n,m,r,nsub,alpha,beta", CASES)
def test_quadratic_increment_matches_oracle(lri, oracle, n, m, r, nsub, alpha, beta, precision, tol):
    U, S, V, nu, dt = problem(n, m, r, alpha, beta)
    alg = lambda k: k.RankAdaptiveUnconventionalAlgorithm(1e-8, rmax=r, K_alg=k.RK4(nsub), rmin=r)

    def exact(a, b):
        prob = oracle.MatrixDEProblem(oracle.BurgersOp(n, 1.0, nu, alpha=a, beta=b),
                                      oracle.SVDLikeRepresentation(U, S, V), (0.0, dt))
        return oracle.solve(prob, alg(oracle), dt).Y[-1].full()

    Y = exact(alpha, beta)
    Q = Y - exact(0.0, 0.0)
    q = np.linalg.norm(Q)
    assert q >= 0.1 * np.linalg.norm(Y)
    prob = lri.MatrixDEProblem(lri.BurgersOperator(1.0, nu, alpha=alpha, beta=beta), lri.SVDLikeRepresentation(U, S, V),
                               (0.0, dt))
    y = lri.solve_burgers_large(prob, alg(lri), dt, precision=precision).Y[-1]
    err = y.full() - Y
    assert np.linalg.norm(err) <= tol * q
    assert abs(np.sum(err * Q)) <= (5e-7 if precision == "fp32" else tol) * q * q
