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
