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
    (10000, 50, 0, 0, 1), (10000, 100, 0, 0, 0), (3000, 60, 0, 1, 1), (3000, 60, 0, 0, 0), (3000, 119, 0, 1, 0),
    (1500, 20, 1, 0, 1), (1500, 80, 1, 0, 0), (600, 20, 1, 1, 0), (1000, 20, 1, 1, 1), (1000, 119, 1, 1, 0),
    (1500, 100, 1, 1, 1), (1500, 10, 0, 1, 1)])
def test_staged_recheck(plan, nrows, k, same, fp32, staged):
    assert plan.plan_staged_recheck(nrows, k, same, fp32) == staged


@pytest.mark.parametrize("nrt,slots,nct,smax,best", [
    (5, 304, 3, 8, (3,)), (13, 304, 7, 8, (7, 8)), (22, 304, 11, 8, (6, 8)), (32, 304, 16, 8, (8,)), (32, 152, 16, 8, (4, 8)),
    (44, 304, 22, 8, (6,)), (1, 304, 188, 32, (32,)), (13, 152, 94, 32, (23,))])
def test_segments(plan, nrt, slots, nct, smax, best):
    assert plan.plan_choose_segments(nrt, slots, nct, smax) in best


def test_segments_use_what_there_is(plan):
    """Few tiles: a segment each, whatever share of the device they fill."""
    for nct in range(1, 9):
        for nrt in range(1, 8):
            assert plan.plan_choose_segments(nrt, 304, nct, 8) == nct, (nrt, nct)


@pytest.mark.parametrize("nref,natoms,k,skips", [
    (1000, 60, 20, 0), (1600, 60, 20, 0), (1600, 200, 20, 0), (1600, 400, 20, 1), (1600, 1200, 20, 1), (1600, 1000, 60, 0),
    (1450, 1200, 10, 1), (1450, 1200, 20, 0), (1200, 1200, 10, 0), (1740, 60, 20, 1), (1700, 1000, 60, 1)])
def test_fp32_skips(plan, nref, natoms, k, skips):
    assert plan.plan_fp32_skips(nref, natoms, k) == skips


@pytest.mark.parametrize("n,natoms,k,segs", [(2200, 1200, 20, 2), (1800, 200, 20, 2), (1450, 1200, 10, 3), (2200, 60, 20, 5),
                                             (2000, 1000, 80, 5), (4800, 400, 30, 5), (8000, 400, 20, 5)])
def test_fp32_skip_segments(plan, n, natoms, k, segs):
    """(5 stands for what choose_segments gave)"""
    assert plan.plan_fp32_skip_segments((n + 31) // 32, 152, natoms, k, 5) == segs


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
