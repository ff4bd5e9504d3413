"""The FP32 screen's segments and lists (k_screen_fp32 in csrc/knn_rms.cu): the
pairs are recomputed by the same recheck whichever screen proposed them, so the
answer must equal the tensor-core screen's bit for bit."""
import numpy as np
import pytest

from mdsctk_gb300 import synth

pytestmark = pytest.mark.gpu


# (references, fit frames or None, atoms, k): one row and a tile of 32 and its
# edges (the most segments), K' from 64 (two blocks per SM) to the largest pool
@pytest.mark.parametrize("nref,nfit,atoms,k", [
    (700, 1, 40, 5),
    (5000, 31, 33, 20),
    (5000, 33, 64, 60),
    (2100, 300, 50, 120),
    (900, None, 61, 16),
    (1500, None, 40, 100),
    (1680, None, 40, 20),  # 21 column tiles: no skipping
    (1690, None, 40, 20),  # 22: skipping
    (1300, None, 40, 200),
])
@pytest.mark.parametrize("nofit", [False, True])
def test_fp32_equals_tensor_cores(ctx, nref, nfit, atoms, k, nofit):
    x = synth.trajectory(nref, atoms, seed=nref, basins=5, dwell=90, drift_sigma=0.06)
    y = None if nfit is None else synth.trajectory(nfit, atoms, seed=7, basins=5, dwell=90, drift_sigma=0.06)
    m = synth.uniform_masses(atoms)
    d, i = ctx.knn_rms(x, y, m, k, precision="fp32", nofit=nofit)
    d2, i2 = ctx.knn_rms(x, y, m, k, precision="bf16x3", nofit=nofit)
    assert np.array_equal(d, d2)
    assert np.array_equal(i, i2)
