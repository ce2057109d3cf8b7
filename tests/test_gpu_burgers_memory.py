"""Device memory of a large Burgers engine: FP32 engines, whose flows run in the
flow kernels and on the tensor cores at every rank, hold no buffers of the
per-stage products (3 x 8 splits of a max(n, m) x 2 r_max panel and one more);
FP64 engines and ones without those kernels do, and still step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def engine(lri, precision, n, m, r, beta):
    h = 1.0 / 512
    op = lri.BurgersOperator(h, np.full(m, 0.01), alpha=0.0, beta=beta)
    return lri.BurgersLargeEngine(op, n, m, r, r, 1e-6, lri.RK4(1), r, precision)


def held(lri, *args):
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    eng = engine(lri, *args)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    eng.close()
    return used


def test_fp32_engine_without_stage_buffers(lri):
    n, m, r = 512, 32768, 64
    panel = 4 * m * 2 * r
    held(lri, "fp32", 256, 256, 64, -0.5)  # the kernels' own load
    a = held(lri, "fp32", n, m, r, -0.5)
    b = held(lri, "fp32", n, m // 2, r, -0.5)
    # what grows with the rows of a panel: three work panels, K/L and its stages,
    # bases, tensor partials (128 columns x 1024 rows hold 8256 x 128 sums), ...
    grows = 3 * panel + 4 * panel + 4 * panel + 4 * 8256 * 128 * (m // 1024)
    assert a - b <= grows / 2 + 16e6


@pytest.mark.parametrize("precision,beta,n,m,r", [("fp64", -0.5, 140, 150, 33), ("fp64", -0.5, 140, 150, 20),
                                                  ("fp32", 0.0, 140, 150, 40), ("fp64", 0.0, 140, 150, 40)])
def test_engines_with_stage_flows_step(lri, oracle, precision, beta, n, m, r):
    g = np.random.default_rng(2)
    U, V = (np.linalg.qr(g.standard_normal((k, r)))[0] for k in (n, m))
    Y0 = lri.SVDLikeRepresentation(U, np.diag(2.0 ** (-np.arange(r) / 8.0)), V)
    h, nu, dt = 1.0 / 64, g.uniform(0.005, 0.02, m), 1e-3
    alg = lambda k: k.RankAdaptiveUnconventionalAlgorithm(1e-8, rmax=r, K_alg=k.RK4(1), rmin=r)
    y = lri.solve_burgers_large(lri.MatrixDEProblem(lri.BurgersOperator(h, nu, alpha=0.0, beta=beta), Y0, (0.0, 2 * dt)),
                                alg(lri), dt, precision=precision).Y[-1]
    po = oracle.MatrixDEProblem(oracle.BurgersOp(n, h, nu, alpha=0.0, beta=beta),
                                oracle.SVDLikeRepresentation(Y0.U, Y0.S, Y0.V), (0.0, 2 * dt))
    yo = oracle.solve(po, alg(oracle), dt).Y[-1]
    assert oracle.rel_fro_err(y.full(), yo.full()) <= (1e-10 if precision == "fp64" else 1e-5)
