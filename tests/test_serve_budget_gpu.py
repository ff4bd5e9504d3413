"""A server's slots within its HBM budget: the workspace of the staged recheck
takes no slot away, and a slot without it serves the same results."""
import numpy as np
import pytest

from mdsctk_gb300 import synth


@pytest.mark.gpu
def test_slots_within_the_budget():
    from mdsctk_gb300.serve import Server

    atoms, cap = 40, 4096
    land = synth.trajectory(3000, atoms, seed=5, basins=2, dwell=200)
    q = synth.trajectory(cap, atoms, seed=6, basins=2, dwell=200)
    kw = dict(k=20, sigma=1.0, nev=2, max_batch_frames=cap)
    with Server(land, None, slots=1, **kw) as srv:
        roomy = srv.stats()["slot_bytes"]
        want = srv.wait(srv.submit(q))[:3]
    # per row of a batch: 28 words, 128 candidates of 48 bytes, a row number
    scratch = cap * (28 * 4 + 128 * 48 + 4)
    with Server(land, None, slots=2, hbm_budget=2 * (roomy - scratch), **kw) as srv:
        assert srv.stats()["slots"] == 2
        got = srv.wait(srv.submit(q))[:3]
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
