"""Bounded device waits that run out, in forms that fault or hang nothing
(mds_test_inject): the call reports MDS_ERR_TIMEOUT and the same context then
computes the same result as before."""
import numpy as np
import pytest

from mdsctk_gb300 import _lib as L
from mdsctk_gb300 import synth


def _expect_timeout(ctx, what, call):
    L.check(ctx.h, ctx._lib.mds_test_inject(ctx.h, what))
    with pytest.raises(L.MdsError) as e:
        call()
    assert e.value.code == L.MDS_ERR_TIMEOUT, e.value


@pytest.mark.gpu
@pytest.mark.parametrize("n,atoms", [(8, 20), (100, 200)])
def test_full_matrix_reports_any_warp(ctx, n, atoms):
    """One warp gives up on a chunk that every other warp still gets: the
    rows it leaves out must not be returned as if they were there."""
    x = synth.trajectory(n, atoms, seed=n)
    m = synth.uniform_masses(atoms)
    d0, i0 = ctx.knn_rms(x, None, m, 0, sort=False)
    _expect_timeout(ctx, L.MDS_INJECT_FULL_STALL, lambda: ctx.knn_rms(x, None, m, 0, sort=False))
    d1, i1 = ctx.knn_rms(x, None, m, 0, sort=False)
    assert np.array_equal(d0, d1) and np.array_equal(i0, i1)


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [100, 5000])  # one K-block of a row, and more than the pipeline's stages
def test_binary_product_times_out(ctx, dim):
    r = np.random.default_rng(dim)
    idx = np.sort(np.stack([r.choice(dim, 20, replace=False) for _ in range(2300)]), axis=1).astype(np.int32)
    a = (np.arange(2301, dtype=np.int64) * 20, idx.ravel(), np.ones(idx.size))
    d0, i0 = ctx.knn_data_sparse(a, None, 12)
    assert ctx.stats()["launches"] == 3
    _expect_timeout(ctx, L.MDS_INJECT_OVERLAP_STALL, lambda: ctx.knn_data_sparse(a, None, 12))
    d1, i1 = ctx.knn_data_sparse(a, None, 12)
    assert np.array_equal(d0, d1) and np.array_equal(i0, i1)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [10, 200])  # the recheck in stages; the block kernel alone
@pytest.mark.parametrize("n", [200, 2000])
def test_no_recheck_of_a_screen_that_timed_out(ctx, n, k):
    """A screen that gave up leaves lists unwritten: whatever they hold, the
    recheck must not follow their indices. Seen from the result arrays, which
    stay as they were."""
    import torch

    x = torch.from_numpy(synth.trajectory(n, 96, seed=90 + n, basins=2, dwell=100)).cuda()
    m = torch.ones(96, device="cuda")
    kk = min(k, n - 1)
    d0, i0 = (t.clone() for t in ctx.knn_rms(x, None, m, k, precision="bf16x3"))
    out = (torch.full((n, kk), -7.0, dtype=torch.float64, device="cuda"),
           torch.full((n, kk), -7, dtype=torch.int32, device="cuda"))
    # (skip=False: no pivot pass, which would take the fault)
    call = lambda: ctx.knn_rms(x, None, m, k, precision="bf16x3", out=out, skip=False)
    torch.cuda.synchronize()
    _expect_timeout(ctx, L.MDS_INJECT_SCREEN_STALL, call)
    assert bool((out[0] == -7).all()) and bool((out[1] == -7).all())
    d1, i1 = call()
    assert torch.equal(d0, d1) and torch.equal(i0, i1)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [150, 3000])  # two clusters of blocks; most of the device
def test_lanczos_cycle_times_out(ctx, n):
    r = np.random.default_rng(n)
    p = r.uniform(size=(n, 2))
    d, i = ctx.knn_data(p, None, 10)
    g = ctx.sysparse(d, i)
    call = lambda: ctx.decomp_sparse(*g, 0.3, 4)
    e0, v0, _, _ = call()
    _expect_timeout(ctx, L.MDS_INJECT_LANCZOS_STALL, call)
    e1, v1, _, _ = call()
    assert np.array_equal(e0, e1) and np.array_equal(v0, v1)
