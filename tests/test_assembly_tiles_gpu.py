"""make_sysparse / make_gesparse at the edges of the assembly's tiles (4,096
list entries, 4,096 keys per sort tile): one entry, one less and one more
than a tile, several tiles with a remainder; lists with repeated edges, self
edges and indices outside the matrix. Bit-identical to the oracle, which
restates the reference's put / cursor semantics directly."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["sys", "ge", "ge_sym"])
@pytest.mark.parametrize("n,maxk,k", [(1, 1, 1), (585, 7, 7), (4096, 1, 1), (1024, 4, 4), (4097, 1, 1), (2731, 5, 3),
                                      (3000, 11, 11)])
def test_assembly_at_tile_edges(ctx, oracle, mode, n, maxk, k):
    rng = np.random.default_rng(n + maxk)
    idx = rng.integers(0, n, size=(n, maxk)).astype(np.int32)
    near = (np.arange(n)[:, None] + rng.integers(-3, 4, size=(n, maxk))) % n
    idx = np.where(rng.random((n, maxk)) < 0.6, near, idx).astype(np.int32)  # many edges listed by both ends
    dist = rng.uniform(0, 2, size=(n, maxk))
    if mode == "sys":
        a, b = ctx.sysparse(dist, idx, k), oracle.sysparse(dist, idx, k)
    else:
        sym = mode == "ge_sym"
        a, b = ctx.gesparse(dist, idx, k, symmetric=sym), oracle.gesparse(dist, idx, k, symmetric=sym)
    for u, v in zip(a[1:], b[1:]):
        assert np.array_equal(u, v)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["sys", "ge", "ge_sym"])
def test_assembly_indices_outside(ctx, oracle, mode):
    """Neighbours past the last row: no column of theirs (and for the
    symmetric general form their transposed entries) is written, nor any
    column at all once a key's column is negative."""
    rng = np.random.default_rng(9)
    for low in (0, -2):
        idx = rng.integers(low, 1500, size=(1000, 6)).astype(np.int32)
        dist = rng.uniform(0, 2, size=idx.shape)
        if mode == "sys":
            a, b = ctx.sysparse(dist, idx), oracle.sysparse(dist, idx)
        else:
            a = ctx.gesparse(dist, idx, symmetric=mode == "ge_sym")
            b = oracle.gesparse(dist, idx, symmetric=mode == "ge_sym")
        for u, v in zip(a[1:], b[1:]):
            assert np.array_equal(u, v)
