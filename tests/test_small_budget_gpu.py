"""knn_rms within an HBM budget that holds the frames, their deviations, one
candidate list per row and the result, but not the workspaces of the faster
paths: the call runs with less and returns the same result."""
import numpy as np
import pytest

from mdsctk_gb300 import Context, synth


def _least(n_ref, n_fit, atoms, width, kprime):
    """Bytes of what no path can do without: frames, deviations (rows of 64
    atoms), records, U, the result, a list of keys per row, the flagged rows."""
    ap = (atoms + 63) // 64 * 64
    fit = n_fit or n_ref
    per = 12 * atoms + 12 * ap + 64
    return n_ref * (per + 80) + (n_fit * per if n_fit else 0) + fit * (12 * width + 8 * kprime + 4 + 4 + 4)


@pytest.mark.gpu
@pytest.mark.parametrize("n_ref,n_fit,atoms,k,precision,kprime", [
    (4000, 0, 100, 20, "fp32", 64), (8000, 40, 100, 20, "fp32", 64), (8000, 0, 100, 20, "fp32", 64),
    (8000, 500, 100, 20, "bf16x3", 512), (8000, 0, 100, 20, "bf16x3", 512)])
def test_same_result_with_less(n_ref, n_fit, atoms, k, precision, kprime):
    x = synth.trajectory(n_ref, atoms, seed=3, basins=4, dwell=200)
    f = synth.trajectory(n_fit, atoms, seed=4, basins=4, dwell=200) if n_fit else None
    with Context(0) as c:
        d0, i0 = c.knn_rms(x, f, None, k, precision=precision)
    least = _least(n_ref, n_fit, atoms, k, kprime)
    if precision == "bf16x3":  # the split operands: 128 (row) and 240 (column) rows of hi|lo per 40 and 80 frames
        ap = (atoms + 63) // 64 * 64
        least += ((n_fit or n_ref) // 40 + 1) * 128 * 4 * ap + (n_ref // 80 + 1) * 240 * 4 * ap
    with Context(0, hbm_budget=least + (256 << 10)) as c:
        d1, i1 = c.knn_rms(x, f, None, k, precision=precision)
    assert np.array_equal(d0, d1) and np.array_equal(i0, i1)


@pytest.mark.gpu
def test_full_matrix_with_less():
    n, atoms = 1500, 100
    x = synth.trajectory(n, atoms, seed=3, basins=4, dwell=200)
    with Context(0) as c:
        d0, i0 = c.knn_rms(x, None, None, 0, sort=False)
    with Context(0, hbm_budget=_least(n, 0, atoms, n, 0) + (80 << 10)) as c:
        d1, i1 = c.knn_rms(x, None, None, 0, sort=False)
    assert np.array_equal(d0, d1) and np.array_equal(i0, i1)
