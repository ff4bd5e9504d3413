"""knn_data_sparse on binary vectors through the tensor-core product: sizes
that fill no tile (128 x 256 pairs, 128 indices), rows past one staged chunk
(65,536 indices), selections read from shared and from global memory, ranges
of values wider than one histogram, overlaps far above 2^11 and 2^14 (where an
accumulator of fewer than 24 bits would round), ties at every rank, and rows
that only look binary. Distances are square roots of integers: equality, and
index order among equal distances, exactly. The integers are counted on the
CPU (sums of 0/1 below 2^24, exact in FP32). contact_profile's masks at grids that fill no word, and groups past
the staged atoms."""
import numpy as np
import pytest


def _csr(rows):
    off = np.zeros(len(rows) + 1, np.int64)
    off[1:] = np.cumsum([len(r) for r in rows])
    idx = np.concatenate(rows).astype(np.int32) if len(rows) else np.zeros(0, np.int32)
    return off, idx, np.ones(len(idx))


def _expect(fit, ref, k):
    d2 = fit.sum(1)[:, None] + ref.sum(1)[None, :] - 2 * (fit.astype(np.float32) @ ref.T.astype(np.float32)).astype(np.int64)
    order = np.argsort(d2, axis=1, kind="stable")[:, 1:k + 1]
    return np.sqrt(np.take_along_axis(d2, order, 1).astype(np.float64)), order


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,dim,density,k", [
    (2305, 0, 127, 0.3, 5), (2560, 0, 128, 0.5, 1), (2400, 0, 1000, 0.02, 33), (25000, 300, 300, 0.4, 7),
    (40001, 140, 130, 0.5, 40), (2300, 2299, 20001, 0.9, 12), (2500, 0, 70001, 0.001, 9), (30011, 257, 513, 0.0, 3)])
def test_overlap_exact(ctx, n, m, dim, density, k):
    rng = np.random.default_rng(dim + n)
    a = rng.random((n, dim)) < density * rng.uniform(0.2, 1.1, size=(n, 1))
    a[::7] = a[1::7][:len(a[::7])] if len(a[1::7]) >= len(a[::7]) else a[::7]  # repeated rows: ties at zero
    a[3] = False
    a[:, -1] = True if density else a[:, -1]  # (the last index is used: the rows' width is dim)
    if not density:
        a[5, dim - 1] = True  # all rows but one are empty: every rank is a tie
    b = a if not m else rng.random((m, dim)) < density * 1.05
    if m and density:
        b[0] = a[17]
    rows = lambda x: [np.flatnonzero(r) for r in x]  # noqa: E731
    d, i = ctx.knn_data_sparse(_csr(rows(a)), _csr(rows(b)) if m else None, k)
    assert ctx.stats()["launches"] >= 3  # byte rows, product, selection
    ed, ei = _expect(b, a, k)
    assert np.array_equal(d, ed)
    assert np.array_equal(i, ei)


@pytest.mark.gpu
@pytest.mark.parametrize("spoil", ["value", "order", "negative", "repeat"])
def test_rows_that_are_not_binary(ctx, oracle, spoil):
    """One entry of one late row is off: the call takes the exact walk."""
    rng = np.random.default_rng(4)
    n, dim = 2400, 60
    off, idx, val = _csr([np.flatnonzero(r) for r in rng.random((n, dim)) < 0.1])
    e = int(off[2000])
    assert off[2001] - off[2000] >= 3
    if spoil == "value":
        val[e + 1] = 0.5
    elif spoil == "order":
        idx[e], idx[e + 1] = idx[e + 1], idx[e]
    elif spoil == "negative":
        idx[e] = -3
    else:
        idx[e + 1] = idx[e]
    fit = tuple(x.copy() for x in (off[1990:2011] - off[1990], idx[off[1990]:off[2010]], val[off[1990]:off[2010]]))
    d, i = ctx.knn_data_sparse((off, idx, val), fit, 6)
    od, oi = oracle.knn_data_sparse((off, idx, val), fit, 6)
    assert np.array_equal(d, od)
    d, i = ctx.knn_data_sparse((off, idx, val), None, 6)
    od, oi = oracle.knn_data_sparse((off, idx, val), None, 6)
    assert np.array_equal(d, od)


@pytest.mark.gpu
@pytest.mark.parametrize("n1,n2,na", [(1, 1, 2), (1, 33, 40), (33, 1, 40), (7, 9, 20), (31, 257, 300), (300, 5, 310),
                                      (1100, 1000, 2100)])
def test_contact_masks(ctx, oracle, n1, n2, na):
    rng = np.random.default_rng(n1 * n2)
    x = rng.uniform(0, 2.5, size=(5, na, 3)).astype(np.float32)
    x[2] = 0.0  # every pair in contact
    x[3] = np.arange(na)[:, None] * 10.0  # none
    g1 = rng.permutation(na)[:n1].astype(np.int32)
    g2 = rng.permutation(na)[:n2].astype(np.int32)
    off, idx = ctx.contact_profile(x, g1, g2, 9.0)
    ooff, oidx = oracle.contact_profile(x, g1, g2, 9.0)
    assert np.array_equal(off, ooff) and np.array_equal(idx, oidx)
