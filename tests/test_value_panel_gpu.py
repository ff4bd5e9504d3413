"""The FP32 vector screen through panels of values (k_dot_panel and
k_panel_select in csrc/knn_data.cu) against the FP64 oracle. The distances are
recomputed in the reference's arithmetic, so they are compared bit for bit; the
indices may differ among exactly equal distances only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(d, i, od, oi):
    assert np.array_equal(d, od)
    for r, c in np.argwhere(i != oi):
        assert np.sum(od[r] == od[r, c]) >= 2 or od[r, c] == od[r, -1]


# (references, fit rows or None, dimension, k): a tile of one row and column
# and their edges (64 x 128); dimensions around the vector loads (4) and the
# staged chunks (32); K' = 64 and 96 (pools of 256 keys), 128 and 192 (512);
# one fit row (several segments) and many
SHAPES = [
    (127, 63, 1, 1),
    (128, 64, 4, 5),
    (129, 65, 33, 9),
    (2000, None, 31, 20),
    (1111, 1, 64, 40),
    (20_011, 3, 50, 20),
    (5003, 700, 97, 63),
    (3000, 200, 8, 64),
    (4001, 130, 5, 126),
]


@pytest.mark.parametrize("corr", [False, True])
@pytest.mark.parametrize("nref,nfit,dim,k", SHAPES)
def test_panel_shapes(ctx, oracle, nref, nfit, dim, k, corr):
    if corr and dim < 4:
        dim = 4  # (two vectors of one component have no correlation)
    rng = np.random.default_rng(nref + dim)
    ref = rng.normal(size=(nref, dim))
    fit = None if nfit is None else rng.normal(size=(nfit, dim))
    d, i = ctx.knn_data(ref, fit, k, correlation=corr)
    _check(d, i, *oracle.knn_data(ref, fit, k, correlation=corr))


@pytest.mark.parametrize("distinct", [1, 7, 300])
def test_panel_ties(ctx, oracle, distinct):
    """More exactly equal values than a list holds: the thinning drops ties,
    the row is then rechecked against every reference."""
    rng = np.random.default_rng(distinct)
    ref = rng.normal(size=(distinct, 12))[rng.integers(0, distinct, size=3000)]
    fit = rng.normal(size=(90, 12))
    d, i = ctx.knn_data(ref, fit, 15)
    _check(d, i, *oracle.knn_data(ref, fit, 15))


def test_several_panels(ctx, oracle):
    """17,000 x 17,000 values take more than one panel of 1 GiB."""
    x = np.random.default_rng(2).normal(size=(17_000, 6))
    d, i = ctx.knn_data(x, None, 12)
    assert ctx.stats()["screen_launches"] == 2
    rows = np.r_[0:40, 15_600:15_800, 16_960:17_000]
    _check(d[rows], i[rows], *oracle.knn_data(x, x[rows], 12))


def test_without_room_for_a_panel(oracle):
    """A budget below the panel's size: the screen that keeps its lists in
    shared memory, the same answer."""
    from mdsctk_gb300 import Context

    x = np.random.default_rng(3).normal(size=(3000, 16))
    with Context(0, hbm_budget=24 << 20) as c:
        d, i = c.knn_data(x, None, 10)
        assert c.stats()["screen_launches"] == 1
    _check(d, i, *oracle.knn_data(x, None, 10))
