"""Device buffers of a batch that the caller replaced by its own: upload and
the steps use them (also larger ones), and the batch's own stay untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def instance(g, n, m, r):
    A = (g.uniform(0.5, 1, n), -2 - g.uniform(0, 1, n), g.uniform(0.5, 1, n))
    B = (g.uniform(0.5, 1, m), -2 - g.uniform(0, 1, m), g.uniform(0.5, 1, m))
    U, V = (np.linalg.qr(g.standard_normal((k, r)))[0] for k in (n, m))
    return A, B, U, np.diag(2.0 ** -np.arange(1.0, r + 1)), V


@pytest.mark.parametrize("precision", ["fp64", "fp32", "df"])
@pytest.mark.parametrize("names", [("U",), ("S", "V"), ("opA", "opB"), ("U", "S", "V", "opA", "opB")])
def test_upload_into_replaced_buffers(lri, names, precision):
    import torch
    g = np.random.default_rng(4)
    shapes = [(33, 31, 3), (64, 40, 5)]
    ins = [instance(g, *s) for s in shapes]
    factors = [lri.SVDLikeRepresentation(U, S, V) for _, _, U, S, V in ins]
    ops = [lri.SylvesterTridiagOperator(A, B) for A, B, _, _, _ in ins]

    def batch():
        return lri.Batch(*(list(x) for x in zip(*shapes)), lri.UnconventionalAlgorithm(lri.RK4(1)),
                         lri._native.LRI_OP_SYLVESTER_TRIDIAG, precision)

    ref, b = batch(), batch()
    own = {k: getattr(b, k) for k in names}
    for k in names:
        setattr(b, k, torch.full((own[k].numel() + 7,), 3.0, dtype=own[k].dtype, device=own[k].device))
    for x in (ref, b):
        x.upload(factors, ops)
        x.step(0.0, 1e-2, 2)
        x.check_status()
    for y, z in zip(ref.download(), b.download()):
        assert np.array_equal(y.U, z.U) and np.array_equal(y.S, z.S) and np.array_equal(y.V, z.V)
    for x in own.values():
        assert not x.any()
    ref.close()
    b.close()
