"""The two-band row and column kernels (FFT mode 1) where their noise cut-off
and sign handling can go wrong, against the 2D-transform path (mode 0) of the
same engine: beams with negative lobes (all four sign components, wrapped
rows and columns), noise that cuts most columns, and datasets of one beam set
whose cut-offs differ.  Tolerances as between the two paths elsewhere: P(D)
within 1e-10 of its peak, log-likelihood within 1e-7, status codes equal;
splits equal or both at the bottom of the
marginal (below 1e-9 of its peak, as in the full-size tests)."""
import numpy as np
import pytest

from test_gpu_2d import _beam2d, spec2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,noise,neg", [
    (512, [(0.0025, 0.003)], True),
    (512, [(0.012, 0.02)], False),
    (1024, [(0.0025, 0.003)], True),
    (1024, [(0.0025, 0.003), (0.008, 0.011)], False),
    (2048, [(0.003, 0.0035), (0.0025, 0.012), (0.01, 0.003)], False),
])
def test_row_and_column_kernels_match_2d_path(gpu_ctx, beams, n, noise, neg):
    from pofd_affine_b200 import calcLikeDouble, doublebeam, synth
    kw = dict(beams_pair=(_beam2d(beams, "band12_0"), _beam2d(beams, "band12_1")), ps=8.0,
              minval=1e-7, nh=30) if neg else {}
    s = spec2(n=n, nedge=96, shape=(64, 64), ndata=len(noise), **kw)
    G = calcLikeDouble(gpu_ctx, s["kp"], s["sk"], s["ok"], n, 96, True, s["nbins"])
    G.addBeamSet(doublebeam(s["b1"], s["b2"], s["ps"], True, s["nh"], s["minval"]))
    for (m1, m2), (s1, s2) in zip(s["maps"], noise):
        G.addDataset(0, m1, m2, s1, s2)
    G.setRRanges(s["th"])
    th = synth.proposals(s["th"], 3, 0.02, rng=1)
    th[:, -2:] = [[1.0, 1.0], [1.1, 0.9], [0.95, 1.05]]
    res = []
    for mode in (1, 0):
        G.setFFT(mode)
        assert G.fusedColumns() == (mode == 1)
        ll, st = G.getLogLikeBatch(th)
        res.append((ll, st, [G.getPD(0, d, th[1], setLog=False) for d in range(len(noise))]))
    (l1, s1, p1), (l0, s0, p0) = res
    assert list(s1) == list(s0) == [0, 0, 0]
    assert np.max(np.abs(l1 - l0)) < 1e-7
    for (pa, ia), (pb, ib) in zip(p1, p0):
        # the wrapped arrays, each rotated back by its own split
        wa, wb = (np.roll(p, (int(i["split1"]), int(i["split2"])), (0, 1))
                  for p, i in ((pa, ia), (pb, ib)))
        assert np.max(np.abs(wa - wb)) <= 1e-10 * wb.max()
        for k, axis in (("split1", 1), ("split2", 0)):
            # the flat minimum of a marginal decides a split by rounding: any
            # two such splits lie together at its bottom
            lo, hi = sorted((int(ia[k]), int(ib[k])))
            marg = wb.sum(axis)
            assert np.all(marg[lo:hi] < 1e-9 * marg.max())
