"""The tensor-core product of binary vectors over its whole range: overlaps up
to the widest rows that it takes (exact integers in FP32 accumulators), more
than one panel of rows, and which of the two binary paths a set takes, by its
launches: a row pass per set, and a product and a selection per panel, against
a bit pass per set and one popcount kernel."""
import numpy as np
import pytest


def _rows(n, dim, nnz, dense, seed):
    r = np.random.default_rng(seed)
    rows = [dense[i] if i in dense else np.unique(r.integers(0, dim, nnz)) for i in range(n)]
    off = np.concatenate([[0], np.cumsum([len(a) for a in rows])]).astype(np.int64)
    return off, np.concatenate(rows).astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("n,dim,ndense", [(2300, (1 << 20) + 1, 12), (1601, 10_000_003, 6)])
def test_overlaps_up_to_the_widest_rows(ctx, n, dim, ndense):
    """Dense rows of which pairs overlap in 2^13 up to nearly dim indices, odd
    numbers among them, in a set of nearly empty rows."""
    r = np.random.default_rng(dim)
    k = ndense + 3
    dense = {}
    for t in range(ndense):  # sizes from dim / 128 to dim, less a few indices each
        size = dim >> (7 * (ndense - 1 - t) // (ndense - 1))
        a = np.ones(size, bool)
        a[r.integers(0, size, 7 + 5 * t)] = False
        dense[97 * t + 11] = np.flatnonzero(a)
    off, idx = _rows(n, dim, 5, dense, 7)
    d, i = ctx.knn_data_sparse((off, idx, np.ones(len(idx))), None, k)
    assert ctx.stats()["launches"] == 3  # the tensor-core product
    count = np.diff(off)
    top = 0
    for q in dense:
        mask = np.zeros(dim, np.int8)
        mask[dense[q]] = 1
        hit = mask[idx]
        both = np.add.reduceat(hit, off[:-1], dtype=np.int64)
        d2 = count[q] + count - 2 * both
        order = np.argsort(d2, kind="stable")[1:k + 1]
        assert np.array_equal(d[q], np.sqrt(d2[order].astype(np.float64))), q
        assert np.array_equal(i[q], order), q
        both[q] = 0
        top = max(top, int(both.max()))
    assert top > dim // 2 - 1000


@pytest.mark.gpu
def test_two_panels(ctx):
    n, dim, k = 17000, 700, 20  # 2^28 values: 15,616 rows of 17,152, then 1,384
    off, idx = _rows(n, dim, 12, {}, 5)
    d, i = ctx.knn_data_sparse((off, idx, np.ones(len(idx))), None, k)
    assert ctx.stats()["launches"] == 1 + 2 * 2
    x = np.zeros((n, dim), np.float32)
    x[np.repeat(np.arange(n), np.diff(off)), idx] = 1
    rows = np.r_[0:3, 15600:15640, n - 70:n]
    c = x.sum(1)
    d2 = (c[rows][:, None] + c[None] - 2 * (x[rows] @ x.T)).astype(np.int64)
    order = np.argsort(d2, axis=1, kind="stable")[:, 1:k + 1]
    assert np.array_equal(d[rows], np.sqrt(np.take_along_axis(d2, order, 1).astype(np.float64)))
    assert np.array_equal(i[rows], order)


@pytest.mark.gpu
@pytest.mark.parametrize("n_ref,n_fit,launches", [(1601, 0, 3), (2300, 2299, 4), (300, 0, 2), (300, 200, 3),
                                                  (30000, 100, 4)])
def test_which_path(ctx, n_ref, n_fit, launches):
    """152 SMs: the product from 76 tiles of 128 x 256 pairs."""
    off, idx = _rows(n_ref, 500, 20, {}, 3)
    fit = None
    if n_fit:
        fo, fi = _rows(n_fit, 500, 20, {}, 4)
        fit = (fo, fi, np.ones(len(fi)))
    ctx.knn_data_sparse((off, idx, np.ones(len(idx))), fit, 5)
    assert ctx.stats()["launches"] == launches
