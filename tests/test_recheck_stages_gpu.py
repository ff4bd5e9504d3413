"""The staged recheck and the full-matrix kernel of knn_rms at their edges:
k + 1 around the largest that the stages take (120) and around the candidate
capacity (128), rows and atoms that fill no block or staged chunk, fewer
references than candidates, crowded frames (many equal distances, lists past
what a row holds), a separate fit set, no superposition. The staged values are
the block kernel's own sums, so rows of the two paths agree bit for bit: the
same frames asked for with k above the limit (block kernel) start with the same
neighbours. The oracle (FP64) to 1e-4 A as everywhere."""
import numpy as np
import pytest

from mdsctk_gb300 import synth


def _frames(n, na, seed, crowd=False):
    x = synth.trajectory(n, na, seed=seed, basins=3, dwell=60, drift_sigma=0.05)
    if crowd:  # clusters of identical frames, larger than a row's candidate list
        x[: n // 2] = x[np.repeat(np.arange(0, n // 2, 200), 200)[: n // 2]]
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
@pytest.mark.parametrize("n,m,na,k,nofit", [(700, 0, 30, 1, False), (641, 0, 65, 100, False), (900, 0, 64, 118, False),
                                            (900, 0, 64, 119, False), (130, 0, 20, 119, False), (90, 0, 33, 119, False),
                                            (1500, 37, 129, 50, False), (1200, 0, 40, 20, True)])
def test_stages_against_block_kernel(ctx, oracle, precision, n, m, na, k, nofit):
    x = _frames(n, na, n + k)
    q = _frames(m, na, 5) if m else None
    mass = np.linspace(1, 16, na).astype(np.float32)
    d, i = ctx.knn_rms(x, q, mass, k, precision=precision, nofit=nofit)
    od, oi = oracle.knn_rms(x, q, mass, k, nofit=nofit)
    assert np.max(np.abs(d - od)) <= 1e-4
    big = min(n - 1, 150)
    d2, i2 = ctx.knn_rms(x, q, mass, big, precision=precision, nofit=nofit)
    w = min(d.shape[1], big)
    assert np.array_equal(d[:, :w], d2[:, :w]) and np.array_equal(i[:, :w], i2[:, :w])


@pytest.mark.gpu
def test_stages_crowded(ctx, oracle):
    x = _frames(2000, 50, 3, crowd=True)
    d, i = ctx.knn_rms(x, None, None, 60, precision="bf16x3")
    od, _ = oracle.knn_rms(x, None, np.ones(50, np.float32), 60)
    assert np.max(np.abs(d - od)) <= 1e-4
    d2, i2 = ctx.knn_rms(x, None, None, 60, precision="fp32")
    assert np.array_equal(d, d2)
    for r, c in np.argwhere(i != i2):  # (which of more equal frames than a list holds come first is the screens')
        assert np.sum(d[r] == d[r, c]) >= 2 or c == 59


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,na,nofit", [(1, 0, 3, False), (7, 0, 64, False), (8, 16, 65, False), (17, 9, 128, False),
                                          (333, 0, 257, False), (41, 1000, 31, True)])
def test_full_matrix(ctx, oracle, n, m, na, nofit):
    x = _frames(n, na, 8)
    q = _frames(m, na, 9) if m else None
    mass = np.linspace(1, 16, na).astype(np.float32)
    d, i = ctx.knn_rms(x, q, mass, 0, sort=False, nofit=nofit)
    od, _ = oracle.knn_rms(x, q, mass, 0, sort=False, nofit=nofit)
    assert np.max(np.abs(d - od)) <= 1e-4
    assert np.array_equal(i, np.tile(np.arange(n, dtype=np.int32), (m or n, 1)))
    if not m and n > 20:  # the sorted call's values (staged recheck) are the matrix's
        ds, idx = ctx.knn_rms(x, None, mass, 15, nofit=nofit)
        assert np.array_equal(ds, np.take_along_axis(d, idx.astype(np.int64), 1))
