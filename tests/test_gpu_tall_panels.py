"""One step of instances whose panels have millions of entries (the QR of the
instance engine in global memory, column ends beyond 2^21): every row of the
factors against the oracle, at heights where an FP32 estimate of the column
is off by one at the columns' first or last entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def instance(seed, n, m, r):
    g = np.random.default_rng(seed)
    A = (g.uniform(0.5, 1, n), -2 - g.uniform(0, 1, n), g.uniform(0.5, 1, n))
    B = (g.uniform(0.5, 1, m), -2 - g.uniform(0, 1, m), g.uniform(0.5, 1, m))
    U, V = (np.linalg.qr(g.standard_normal((k, r)))[0] for k in (n, m))
    return A, B, U, np.diag(2.0 ** (-np.arange(1, r + 1) / 4.0)), V


def run(module, op, alg, ins, precision=None):
    A, B, U, S, V = ins
    prob = module.MatrixDEProblem(op(A, B), module.SVDLikeRepresentation(U, S, V), (0.0, 1e-2))
    return module.solve(prob, alg, 1e-2, **({"precision": precision} if precision else {})).Y[-1]


def rows_close(a, b, tol):
    return np.linalg.norm(a - b, axis=1).max() <= tol * np.linalg.norm(b, axis=1).max()


# factors: rounding 1e-16 times a core's condition 2^(r/4) <= 2^12, N r sums: < 1e-10
@pytest.mark.parametrize("kind,n,m,r", [("ksl", 114050, 64, 48), ("bug", 114050, 64, 48), ("bug", 40, 205162, 32)])
def test_tall_fp64_steps_match_oracle(lri, oracle, kind, n, m, r):
    ins = instance(r + n, n, m, r)
    alg = {"ksl": lambda k: k.ProjectorSplitting(k.PrimalLieTrotter(), k.RK4(1)),
           "bug": lambda k: k.UnconventionalAlgorithm(k.RK4(1))}[kind]
    y = run(lri, lri.SylvesterTridiagOperator, alg(lri), ins, "fp64")
    yo = run(oracle, oracle.SylvesterTridiagOp, alg(oracle), ins)
    for a, b in ((y.U, yo.U), (y.S, yo.S), (y.V, yo.V)):
        assert rows_close(a, b, 1e-10)


# rank-adaptive: the columns' signs are free, so Y's rows; FP32: a row of Q is
# good to about 64 * 2^-24 of the longest
@pytest.mark.parametrize("precision,n,m,r,tol", [("fp64", 107744, 80, 28, 1e-10), ("fp32", 102581, 80, 32, 1e-4)])
def test_tall_rank_adaptive_steps_match_oracle(lri, oracle, precision, n, m, r, tol):
    ins = instance(r + n, n, m, r)
    alg = lambda k: k.RankAdaptiveUnconventionalAlgorithm(1e-9, rmax=r, K_alg=k.RK4(1), rmin=r)
    y = run(lri, lri.SylvesterTridiagOperator, alg(lri), ins, precision)
    yo = run(oracle, oracle.SylvesterTridiagOp, alg(oracle), ins)
    assert y.S.shape == yo.S.shape == (r, r)
    assert rows_close((y.U @ y.S) @ y.V.T, (yo.U @ yo.S) @ yo.V.T, tol)
    assert np.abs(y.U.T @ y.U - np.eye(r)).max() <= (1e-12 if precision == "fp64" else 1e-4)
