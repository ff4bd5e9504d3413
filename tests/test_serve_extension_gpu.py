"""The serving extension at sizes off its warp: a request of one frame, lists
shorter and longer than a warp, more eigenvectors than lanes. Against the file
pipeline's own sums (general matrix of the served lists, kernelised with the
landmark degrees, times z / lambda) restated by the oracle. The kernel sums the
same terms in the same order in FP64; 1e-10 covers exp and the fused
multiply-adds of sums of at most 70 terms of size below 1."""
import numpy as np
import pytest

from mdsctk_gb300 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("k,nev,sizes", [(5, 2, (1, 3)), (32, 33, (1, 129)), (70, 4, (2, 31))])
def test_extension_sizes(ctx, oracle, k, nev, sizes):
    from mdsctk_gb300.serve import Server

    land = synth.trajectory(400, 40, seed=k, basins=2, dwell=80)
    m = synth.uniform_masses(40)
    d, i = oracle.knn_rms(land, None, m, k)
    sigma = float(np.median(d))
    # (the model's degrees come from its own landmark distances, FP32 to 1e-6 A)
    n, pcol, irow, val = oracle.sysparse(*ctx.knn_rms(land, None, m, k, precision="bf16x3"))
    _, dinv = oracle.affinity(n, pcol, irow, val, sigma)
    with Server(land, m, k=k, sigma=sigma, nev=nev, max_batch_frames=256, slots=1) as srv:
        w, V = srv.model()
        for size in sizes:
            q = synth.trajectory(size, 40, seed=100 + size, basins=2, dwell=80)
            ext, dq, iq, _ = srv.wait(srv.submit(q))
            mq, pb, ib, vb = oracle.gesparse(dq, iq)
            b = oracle.affinity_nystrom(mq, pb, ib, vb, sigma, dinv)
            for x in range(nev):
                e = oracle.sp_dgemv(mq, pb, ib, b, V[x] / w[x])
                assert np.max(np.abs(ext[x] - e)) < 1e-10
