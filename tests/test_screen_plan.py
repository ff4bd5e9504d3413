"""The size rules of knn_rms (screen_plan.h), on the CPU, at sizes where both
sides were measured (the figures stand beside the rules); on the GPU, which
path a call takes, by its launches, and the paths' results around the lines."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mdsctk_gb300", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    out = str(tmp_path_factory.mktemp("plan") / "libplan.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC,
                    os.path.join(HERE, "native", "screen_plan_shim.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("nrows,k,same,fp32,staged", [
    (20000, 100, 1, 0, 1), (3000, 20, 1, 0, 1), (100000, 119, 1, 0, 1), (100000, 120, 1, 0, 0), (1000, 50, 1, 0, 0),
    (600, 20, 0, 0, 0), (600, 110, 0, 0, 0), (2047, 20, 0, 0, 1), (2047, 50, 0, 0, 0), (2047, 100, 0, 0, 0),
    (10000, 50, 0, 0, 1), (10000, 100, 0, 0, 0), (3000, 60, 0, 1, 1), (3000, 60, 0, 0, 0), (3000, 119, 0, 1, 0)])
def test_staged_recheck(plan, nrows, k, same, fp32, staged):
    assert plan.plan_staged_recheck(nrows, k, same, fp32) == staged


@pytest.mark.gpu
@pytest.mark.parametrize("n_ref,n_fit,k,extra", [(2000, 600, 110, 0), (1000, 0, 50, 0), (2200, 0, 50, 4), (2200, 0, 119, 4),
                                                 (2200, 2100, 31, 4), (2200, 2100, 32, 0)])
def test_recheck_path(ctx, n_ref, n_fit, k, extra):
    """Against k = 130, which the block kernel takes whatever the size."""
    from mdsctk_gb300 import synth

    x = synth.trajectory(n_ref, 60, seed=1, basins=3, dwell=60)
    f = synth.trajectory(n_fit, 60, seed=2, basins=3, dwell=60) if n_fit else None
    counts = []
    for kk in (k, 130):
        ctx.knn_rms(x, f, None, kk, precision="bf16x3")
        st = ctx.stats()
        assert st["passes"] == 1
        counts.append(st["launches"])
    assert counts[0] == counts[1] + extra


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
@pytest.mark.parametrize("n,m,na,k,nofit,crowd", [
    (2000, 0, 30, 119, False, False), (2001, 0, 65, 118, False, False), (2047, 0, 20, 1, True, False),
    (2600, 0, 33, 100, False, True), (2100, 2005, 40, 31, False, False), (900, 5003, 24, 63, False, True)])
def test_staged_rows_around_the_lines(ctx, oracle, precision, n, m, na, k, nofit, crowd):
    """The staged path's rows against the oracle and, bit for bit, against the
    block kernel's (the same frames asked for with k above the stages' limit)."""
    from mdsctk_gb300 import synth

    x = synth.trajectory(n, na, seed=n + k, basins=3, dwell=60, drift_sigma=0.05)
    if crowd:  # clusters of identical frames, larger than a row's candidate list
        x[: n // 2] = x[np.repeat(np.arange(0, n // 2, 200), 200)[: n // 2]]
    q = synth.trajectory(m, na, seed=5, basins=3, dwell=60, drift_sigma=0.05) if m else None
    mass = np.linspace(1, 16, na).astype(np.float32)
    d, i = ctx.knn_rms(x, q, mass, k, precision=precision, nofit=nofit)
    assert len(d) >= 2000
    d2, i2 = ctx.knn_rms(x, q, mass, 150, precision=precision, nofit=nofit)
    assert np.array_equal(d, d2[:, :k])
    if not crowd:
        assert np.array_equal(i, i2[:, :k])
    rows = np.r_[0:40, len(d) - 40:len(d)]
    od, _ = oracle.knn_rms(x, (x if q is None else q)[rows], mass, k, nofit=nofit)
    assert np.max(np.abs(d[rows] - od)) <= 1e-4
