"""The one-launch Lanczos cycle at its edges: fewer rows than blocks in a
cluster, rows that do not fill a block or a warp's piece, few and many basis
columns, a Krylov space that runs out (ncv = n), a basis that does not fit in
shared memory (60,001 x 120 and 20,011 x 300). Eigenvalues against dense eigh
and every returned pair as an eigenpair of the oracle's operator (for the large
ones, stopped after six restarts: as Ritz pairs, an orthonormal basis with its
Rayleigh quotients and the reported residuals): FP64 with tol = 0 leaves residuals of a few ulps of the
operator's norm 1 per row sum, so 1e-12 covers them with room, and 1e-11 the
eigenvalues of the two solvers and the vectors' orthonormality."""
import numpy as np
import pytest


def _band_graph(n, width, seed):
    """Nodes on a line joined to their `width` successors, distances from the
    seed: a connected graph whose top eigenvalues are simple. (CSC, strict
    lower triangle)."""
    rng = np.random.default_rng(seed)
    cols = np.repeat(np.arange(n), width)
    rows = cols + np.tile(np.arange(1, width + 1), n)
    keep = rows < n
    cols, rows = cols[keep], rows[keep]
    pcol = np.searchsorted(cols, np.arange(n + 1)).astype(np.int32)
    return pcol, rows.astype(np.int32), rng.uniform(0.5, 1.5, size=len(rows))


@pytest.mark.gpu
@pytest.mark.parametrize("n,width,nev,ncv", [(3, 2, 1, 3), (6, 3, 2, 6), (31, 4, 3, 20), (129, 6, 5, 51), (260, 40, 4, 9),
                                             (1000, 20, 10, 0), (4111, 200, 3, 31)])
def test_small_against_dense(ctx, oracle, n, width, nev, ncv):
    pcol, irow, val = _band_graph(n, min(width, n - 1), n)
    w, V, res, nconv = ctx.decomp_sparse(n, pcol, irow, val, 1.0, nev, ncv=ncv)
    assert nconv == nev
    M = oracle.dense_affinity(n, pcol, irow, val, 1.0)
    e = np.linalg.eigvalsh(M)[::-1][:nev]
    assert np.max(np.abs(w - e)) <= 1e-11
    assert np.max(np.abs(V @ M - w[:, None] * V)) <= 1e-12
    assert np.max(np.abs(V @ V.T - np.eye(nev))) <= 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("n,width,nev,ncv", [(60001, 30, 3, 120), (20011, 60, 4, 300)])
def test_basis_past_shared_memory(ctx, oracle, n, width, nev, ncv):
    import scipy.sparse as sp

    pcol, irow, val = _band_graph(n, width, 7)
    sigma = 1.0
    w, V, res, nconv = ctx.decomp_sparse(n, pcol, irow, val, sigma, nev, ncv=ncv, tol=1e-10, maxiter=6)
    L = sp.csc_matrix((np.exp(-val * val / (2 * sigma * sigma)), irow, pcol), shape=(n, n))
    A = L + L.T
    d = 1.0 / np.sqrt(np.asarray(A.sum(axis=1)).ravel())
    A = sp.diags(d) @ A @ sp.diags(d)
    # (the long band's top eigenvalues crowd at 1, so few converge in six
    # restarts: the returned pairs are Ritz pairs of one orthonormal basis)
    R = (A @ V.T).T - w[:, None] * V
    assert np.max(np.abs(V @ V.T - np.eye(nev))) <= 1e-11
    assert np.allclose(np.linalg.norm(R, axis=1) / np.abs(w), res, rtol=1e-6, atol=1e-12)
    assert np.max(np.abs(np.sum(V * (A @ V.T).T, axis=1) - w)) <= 1e-11
