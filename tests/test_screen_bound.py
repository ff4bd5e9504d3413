"""The FP32 screen bound of a frame pair (screen_shifted_f32, qcp.cuh) against
the exact minimum RMSD^2, on the CPU, with the pair's sums rounded from FP64 so
that only the function's own arithmetic is seen.

The screen subtracts a guard of 2^-16 (|a_i|^2 + |a_j|^2) that has to cover the
rounding of the Gram as well. The function itself may take an eighth of it:
D = |a_i|^2 + |a_j|^2 - 2 tr G is three roundings of at most 2 E (E the two
norms' sum, |tr G| <= E / 2) with the three roundings of its inputs, 6 * 2^-24 E;
nu <= D / 2 <= E comes from a quartic whose coefficients and evaluation each
round about a dozen times, 2 nu * 12 * 2^-24 <= 24 * 2^-24 E: together
30 * 2^-24 E < 2^-19 E. Rigid frames (a fluctuation small against the radius
of gyration) are where a start of the root search that cancels shows."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mdsctk_gb300", "csrc")


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    out = str(tmp_path_factory.mktemp("qcp") / "libqcp.so")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC,
                    os.path.join(HERE, "native", "qcp_shim.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


def _superpose(x, mu):
    """x (centred) rotated onto mu (Kabsch)."""
    u, _, vt = np.linalg.svd(np.einsum("nac,ad->ncd", x, mu))
    s = np.sign(np.linalg.det(u @ vt))
    u[:, :, 2] *= s[:, None]
    return x @ (u @ vt)


def _pairs(atoms, rg, sigma, shape, n, seed):
    """Records, Grams and exact RMSD^2 of all pairs of n frames: a chain of the
    given radius of gyration (or a globule of independent atoms) with the
    atoms' fluctuations, superposed onto the first frame in its principal axes,
    as the screen's template is."""
    r = np.random.default_rng(seed)
    c = r.normal(size=(atoms, 3))
    if shape == "chain":
        c = np.cumsum(c, 0)
    c -= c.mean(0)
    c *= rg / np.sqrt((c ** 2).sum(1).mean())
    x = c + sigma * r.normal(size=(n, atoms, 3))
    x -= x.mean(1, keepdims=True)
    x /= np.sqrt(atoms)  # unit total mass
    mu = x[0] @ np.linalg.eigh(x[0].T @ x[0])[1]
    y = _superpose(x, mu)
    a = y - mu
    e = (a ** 2).sum((1, 2))
    U = np.einsum("nac,ad->ncd", a, mu)
    M0 = mu.T @ mu
    sym = 0.5 * (U + U.transpose(0, 2, 1))
    rec = np.zeros((n, 16), np.float32)
    for t, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
        rec[:, t] = M0[i, j] + sym[:, i, j]
        rec[:, 6 + t] = sym[:, i, j]
    rec[:, 12] = U[:, 1, 2] - U[:, 2, 1]
    rec[:, 13] = U[:, 2, 0] - U[:, 0, 2]
    rec[:, 14] = U[:, 0, 1] - U[:, 1, 0]
    rec[:, 15] = e
    iu, ju = np.triu_indices(n, 1)
    G = np.einsum("nac,nad->ncd", a[iu], a[ju])
    S = np.einsum("nac,nad->ncd", y[iu], y[ju])
    w = np.linalg.svd(S, compute_uv=False)
    w[:, 2] *= np.sign(np.linalg.det(S))
    # RMSD^2 from the deviations' scale: |y_i|^2 + |y_j|^2 - 2 sum w, in FP64
    exact = (y[iu] ** 2).sum((1, 2)) + (y[ju] ** 2).sum((1, 2)) - 2.0 * w.sum(1)
    return rec[iu].copy(), rec[ju].copy(), G.reshape(-1, 9).astype(np.float32), exact, e[iu] + e[ju]


@pytest.mark.parametrize("root_ulp", [0, -1, 1])
@pytest.mark.parametrize("refine", [1, 0])
@pytest.mark.parametrize("atoms,rg,sigma,shape", [(58, 1.1, 0.08, "chain"), (60, 1.6, 0.1, "chain"),
                                                  (304, 1.5, 0.08, "chain"), (100, 1.3, 0.05, "chain"),
                                                  (60, 1.6, 0.02, "chain"), (60, 1.6, 0.4, "chain"),
                                                  (60, 1.6, 0.02, "globule"), (304, 1.2, 0.05, "globule")])
def test_bound_stays_below_exact(shim, atoms, rg, sigma, shape, refine, root_ulp):
    rec_i, rec_j, G, exact, E = _pairs(atoms, rg, sigma, shape, 60, atoms + int(100 * sigma))
    out = np.zeros(len(E), np.float32)
    fp = ctypes.POINTER(ctypes.c_float)
    p = [v.ctypes.data_as(fp) for v in (G, rec_i, rec_j)]
    for thr in (np.inf, float(np.median(exact)), 0.0):
        shim.screen_shim(len(E), *p, ctypes.c_float(0.0), ctypes.c_float(thr), refine, root_ulp, out.ctypes.data_as(fp))
        over = (out.astype(np.float64) - exact) / E
        assert over.max() <= 2.0 ** -19, (thr, over.max() * 2 ** 16)
        if refine and thr == np.inf:  # and it is tight: within the guard below the exact value
            assert over.min() >= -2.0 ** -16, over.min() * 2 ** 16


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
@pytest.mark.parametrize("n,atoms,rg,sigma", [(600, 60, 1.6, 0.02), (2000, 60, 1.6, 0.02), (2000, 304, 1.2, 0.05)])
def test_rigid_frames_keep_the_margin(ctx, n, atoms, rg, sigma, precision):
    """Whole calls on rigid frames: the largest over-estimate of a rechecked
    pair stays below a quarter of the guard, so no row is redone for one. FP32:
    1/8 for the function (above) and 1/12 for the Gram (knn_common.cuh); BF16x3,
    with a guard four times as wide: 1/32 and 1/6."""
    from mdsctk_gb300 import synth

    r = np.random.default_rng(n + atoms)
    c = r.normal(size=(atoms, 3))
    c -= c.mean(0)
    c *= rg / np.sqrt((c ** 2).sum(1).mean())
    x = c + sigma * r.normal(size=(n, atoms, 3))
    x = np.einsum("nij,naj->nai", synth._random_rotations(n, r), x) + r.uniform(0, 5, size=(n, 1, 3))
    d, _ = ctx.knn_rms(x.astype(np.float32), None, None, 20, precision=precision)
    st = ctx.stats()
    assert np.isfinite(d).all()
    assert st["screen_err_max"] < 0.25 * st["guard_coef"], st
    assert st["guard_violations"] == 0, st
