"""Starting thresholds and nearest column tiles of a separate fit set (k_seed_thr
in csrc/knn_rms_tc.cu), at the edges of the tiles (40 rows, 80 columns) and of
k + 1 against whole tiles. skip=False runs without them; both recheck exactly,
so the answers must be the same bit for bit."""
import numpy as np
import pytest

from mdsctk_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref,nfit,k", [
    (320, 1, 79),      # four full tiles, k + 1 = one tile
    (321, 21, 80),     # one frame in the last tile, k + 1 = a tile and one frame
    (399, 40, 159),
    (400, 41, 160),
    (330, 60, 300),    # more than four full tiles needed: no threshold
    (4000, 33, 1),
    (4000, 81, 50),
    (20_000, 500, 100),
])
def test_seeded_screen(ctx, nref, nfit, k):
    x = synth.trajectory(nref + nfit, 50, seed=nref + k, basins=6, dwell=60, drift_sigma=0.05)
    m = synth.uniform_masses(50)
    ref, fit = x[:nref], x[nref:]
    d, i = ctx.knn_rms(ref, fit, m, k, precision="bf16x3")
    d2, i2 = ctx.knn_rms(ref, fit, m, k, precision="bf16x3", skip=False)
    assert np.array_equal(d, d2)
    assert np.array_equal(i, i2)


def test_seeded_copies(ctx, oracle):
    """Fit frames that are reference frames, and identical reference frames:
    distances of zero and ties at the threshold."""
    x = synth.trajectory(200, 30, seed=5)
    ref = np.concatenate([x, x, x])
    m = synth.uniform_masses(30)
    d, i = ctx.knn_rms(ref, x[:70], m, 5, precision="bf16x3")
    od, oi = oracle.knn_rms(ref, x[:70], m, 5)
    assert np.max(np.abs(d - od)) <= 1e-4  # the bound of the other tests against the oracle


@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
@pytest.mark.parametrize("k", [10, 80])
def test_rows_with_overfull_lists(ctx, oracle, precision, k):
    """Fit frames about as far from every reference frame as from any other:
    the segments' lists hold more keys below the threshold than a row's buffer
    in the recheck (512), which then keeps its K' smallest."""
    ref = synth.trajectory(6000, 40, seed=3, basins=5, dwell=60)
    fit = np.zeros((45, 40, 3), np.float32)
    fit[20:] = ref[:25] + np.random.default_rng(4).normal(scale=0.6, size=(25, 40, 3)).astype(np.float32)
    m = synth.uniform_masses(40)
    d, _ = ctx.knn_rms(ref, fit, m, k, precision=precision)
    od, _ = oracle.knn_rms(ref, fit, m, k)
    assert np.all(np.diff(d, axis=1) >= 0)
    assert np.max(np.abs(d - od)) <= 1e-4  # the bound of the other tests against the oracle
