"""contact_profile where the masks of all frames do not fit beside the result:
they are made for a batch of frames at a time, the last one a remainder, and
the result has the memory first."""
import numpy as np
import pytest

from mdsctk_gb300 import Context


@pytest.mark.gpu
@pytest.mark.parametrize("eps", [1000.0, 9.0])  # every pair in contact; a few
@pytest.mark.parametrize("spare", [40 << 10, 300 << 10, 1500 << 10, 3 << 20])
def test_masks_in_batches(oracle, eps, spare):
    n, atoms = 1501, 200
    x = np.random.default_rng(0).uniform(0, 3, (n, atoms, 3)).astype(np.float32)
    g1 = np.arange(100, dtype=np.int32)
    g2 = np.arange(100, 193, dtype=np.int32)  # 9,300 pairs: 291 words, 1.75 MB for all frames
    off, idx = oracle.contact_profile(x, g1, g2, eps)
    need = x.nbytes + 4 * len(idx) + 2 * 8 * (n + 1) + 5 * 4096  # (each buffer in whole pages)
    with Context(0, hbm_budget=need + spare) as c:
        goff, gidx = c.contact_profile(x, g1, g2, eps)
    assert np.array_equal(goff, off) and np.array_equal(gidx, idx)
