"""Snapshots sent from the host while steps run, and histories recorded into
one page-locked buffer or into separate ones: exactly the factors of a run that
waits after each step, at odd sizes (parts of a record off 16-byte boundaries),
with the caller's arrays overwritten as soon as a step has returned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32", "df"])
@pytest.mark.parametrize("shapes", [[(33, 31, 3)], [(45, 37, 5), (64, 21, 1), (19, 19, 3)]])
@pytest.mark.parametrize("separate", [False, True])
def test_staged_snapshots_and_records(lri, precision, shapes, separate):
    import torch
    g = np.random.default_rng(5)
    alg = lri.UnconventionalAlgorithm(lri.RK4(1))
    data = [[g.standard_normal((n, m)) for n, m, _ in shapes] for _ in range(7)]
    factors = []
    for (n, m, r), Y in zip(shapes, data[0]):
        U, s, Vt = np.linalg.svd(Y, full_matrices=False)
        factors.append(lri.SVDLikeRepresentation(U[:, :r], np.diag(s[:r]), Vt[:r].T))

    def batch():
        b = lri.Batch([s[0] for s in shapes], [s[1] for s in shapes], [s[2] for s in shapes], alg,
                      lri._native.LRI_OP_DATA, precision)
        b.upload(factors)
        b.data_init(data[0])
        return b

    ref = batch()
    expected = []
    for k in range(1, 7):
        ref.step(0.0, 1.0, 1, data[k])
        torch.cuda.synchronize()
        expected.append(ref.download())
    ref.close()
    b = batch()
    h = lri.History(b, slots=2)
    for k in range(1, 7):
        mine = [Y.copy() for Y in data[k]]
        if k % 2:
            b.step(0.0, 1.0, 1, mine)
        else:
            flat = b.pack_data(mine)
            b.step(0.0, 1.0, 1, np.append(flat, np.zeros(b.Ynext.numel() - flat.size, flat.dtype)))
            flat[:] = np.nan
        for Y in mine:
            Y[:] = np.nan
        host = None
        if separate:
            pin = lambda x, dt: torch.empty(x, dtype=dt, pin_memory=True)
            host = (pin(b.U.numel(), b.dtype), pin(b.S.numel(), b.dtype), pin(b.V.numel(), b.dtype),
                    pin(b.count, torch.int32))
        h.record(host)
    got = h.collect()
    h.close()
    b.check_status()
    b.close()
    for k, (rec, exp) in enumerate(zip(got, expected)):
        for x, y in zip(rec, exp):
            assert np.array_equal(x.U, y.U) and np.array_equal(x.S, y.S) and np.array_equal(x.V, y.V), k
