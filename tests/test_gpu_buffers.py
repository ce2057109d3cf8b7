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


@pytest.mark.parametrize("how", ["no page-locked memory", "too large to stage"])
def test_snapshots_from_pageable_memory(lri, how, monkeypatch):
    import torch
    g = np.random.default_rng(6)
    n, m, r = 45, 37, 5
    data = [g.standard_normal((n, m)) for _ in range(4)]
    U, s, Vt = np.linalg.svd(data[0], full_matrices=False)
    Y0 = lri.SVDLikeRepresentation(U[:, :r], np.diag(s[:r]), Vt[:r].T)

    def run():
        b = lri.Batch([n], [m], [r], lri.UnconventionalAlgorithm(lri.RK4(1)), lri._native.LRI_OP_DATA, "fp64")
        b.upload([Y0])
        b.data_init([data[0]])
        for k in (1, 2, 3):
            mine = data[k].copy()
            b.step(0.0, 1.0, 1, [mine] if k % 2 else mine.ravel(order="F"))
            mine[:] = np.nan
        y = b.download()[0]
        staged = bool(b._stage)
        b.close()
        return y, staged

    ref, staged = run()
    assert staged
    if how == "too large to stage":
        monkeypatch.setattr(lri.Batch, "STAGE_BYTES", 8 * n * m - 1)
    else:
        zeros = torch.zeros

        def refuse(*args, pin_memory=False, **kw):
            if pin_memory:
                raise RuntimeError("CUDA error: out of memory")
            return zeros(*args, **kw)

        monkeypatch.setattr(torch, "zeros", refuse)
    y, staged = run()
    assert not staged
    assert np.array_equal(y.U, ref.U) and np.array_equal(y.S, ref.S) and np.array_equal(y.V, ref.V)


def test_stream_without_the_raw_lookup(lri, monkeypatch):
    import torch
    b = lri.Batch([20], [20], [2], lri.UnconventionalAlgorithm(lri.RK4(1)), lri._native.LRI_OP_ZERO, "fp64")
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        assert b._stream().value == st.cuda_stream
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
        assert b._stream().value == st.cuda_stream
    b.close()


def test_instances_without_a_snapshot_see_zeros(lri):
    """A list shorter than the batch: zeros for the rest, in every step."""
    g = np.random.default_rng(8)
    shapes = [(33, 31, 3), (20, 24, 2)]
    data = [[g.standard_normal(s[:2]) for s in shapes] for _ in range(5)]
    Y0 = [lri.SVDLikeRepresentation(*(lambda U, s, Vt, r: (U[:, :r], np.diag(s[:r]), Vt[:r].T))(
        *np.linalg.svd(Y, full_matrices=False), r)) for Y, (_, _, r) in zip(data[0], shapes)]

    def run(last):
        b = lri.Batch(*(list(x) for x in zip(*shapes)), lri.UnconventionalAlgorithm(lri.RK4(1)),
                      lri._native.LRI_OP_DATA, "fp64")
        b.upload(Y0)
        b.data_init(data[0])
        for k in (1, 2, 3):
            b.step(0.0, 1.0, 1, data[k])
        b.step(0.0, 1.0, 1, last)
        y = b.download()[1]
        b.close()
        return y

    y, ref = run(data[4][:1]), run([data[4][0], np.zeros(shapes[1][:2])])
    assert np.array_equal(y.U, ref.U) and np.array_equal(y.S, ref.S) and np.array_equal(y.V, ref.V)
