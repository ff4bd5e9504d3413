"""knn_data_sparse on sets that look binary but are not: they take the general
walk with the memory that it needs, whatever their first or most values are."""
import numpy as np
import pytest

from mdsctk_gb300 import Context


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["leading_ones", "one_other"])
@pytest.mark.parametrize("separate", [False, True])
def test_not_binary_within_a_small_budget(kind, separate):
    n, dim, nnz, k = 3000, 40000, 40, 10
    r = np.random.default_rng(17)
    idx = np.sort(np.stack([r.choice(dim, nnz, replace=False) for _ in range(n)]), axis=1).astype(np.int32)
    val = np.ones((n, nnz))
    if kind == "leading_ones":
        val[2:] = r.normal(size=(n - 2, nnz))
    else:
        val[5, 1] = 2.0
    off = np.arange(n + 1, dtype=np.int64) * nnz
    a = (off, idx.ravel(), val.ravel())
    fit = (off[:201], idx[:200].ravel(), val[:200].ravel()) if separate else None
    with Context(0) as c:
        d0, i0 = c.knn_data_sparse(a, fit, k)
    # the lists are 1.4 MB (1.7 with a fit set) and the results 0.4; the bit sets 15
    with Context(0, hbm_budget=6 << 20) as c:
        d1, i1 = c.knn_data_sparse(a, fit, k)
    assert np.array_equal(d0, d1) and np.array_equal(i0, i1)
    dense = np.zeros((n, dim), np.float32)
    np.put_along_axis(dense, idx.astype(np.int64), val.astype(np.float32), 1)
    g = (dense @ dense[:20].T).astype(np.float64)
    sq = (val ** 2).sum(1)
    d2 = np.sort(np.maximum(sq[:, None] + sq[None, :20] - 2 * g, 0), axis=0)
    assert np.abs(d1[:20] ** 2 - d2[1:k + 1].T).max() < 1e-3 * sq.max()
