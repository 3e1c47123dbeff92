"""Beams with negative lobes in the single-block kernel: grids with a wrap edge,
whose moments take one value of the grid back while the transform begins.  The
forms that take several datasets of a beam set in turn (512 and 256 threads a
row), a block per dataset, and the mixed sizes on either side of their rule,
against cuFFT's path of the same engine; and every row the same to the last bit
call after call.  Tolerances as between the FFT forms elsewhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(fwhm):
    from pofd_affine_b200 import synth
    g = synth.gaussian_beam(fwhm)
    c = g.shape[0] // 2
    y, x = np.mgrid[0:g.shape[0], 0:g.shape[1]]
    r2 = ((x - c) ** 2 + (y - c) ** 2) / (2.0 * fwhm) ** 2
    return g - 0.05 * r2 * np.exp(1.0 - r2)


@pytest.mark.parametrize("n,ndata,nprop", [
    (1024, 2, 100), (1024, 2, 160), (1024, 3, 9), (2048, 3, 50), (2048, 2, 200),
    (4096, 2, 80), (4096, 3, 150), (8192, 2, 80), (8192, 2, 200),
    (6000, 1, 3), (6000, 2, 74), (6000, 2, 75), (3000, 3, 7)])
def test_wrap_edge(gpu_ctx, n, ndata, nprop):
    from pofd_affine_b200 import beam, calcLike, synth
    rng = np.random.default_rng(n + nprop)
    kp, kv = synth.knot_model(6, 0.002, 0.3, rng=rng)
    bm = _ring(3.0)
    L = calcLike(gpu_ctx, kp, n, 900, True, 300)
    L.addBeamSet(beam(bm, 6.0, True, 100))
    for d in range(ndata):
        s = 0.003 * (1 + 0.3 * d)
        L.addDataset(0, synth.make_map((40, 44 + d), 6.0, bm, kp, kv, 0.001, rng), s)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    L.setRRanges(th0)
    th = synth.proposals(th0, nprop, 0.02, rng=rng)
    out = []
    for mode in (0, 1):
        L.setFFT(mode)
        ll, st = L.getLogLikeBatch(th)
        if mode == 0:
            for _ in range(30):
                l2, s2 = L.getLogLikeBatch(th)
                assert np.array_equal(l2, ll, equal_nan=True) and np.array_equal(s2, st)
        out.append((ll, st, [L.getPD(0, d, th[0], setLog=False) for d in range(ndata)]))
    (l0, s0, p0), (l1, s1, p1) = out
    assert list(s0) == list(s1) and np.all(s1 == 0)
    assert np.all(np.abs(l0 - l1) < 1e-7)
    for (pa, ia), (pb, ib) in zip(p0, p1):
        assert abs(ia["mn"] - ib["mn"]) <= 1e-12 * abs(ib["mn"])
        wa, wb = np.roll(pa, int(ia["splitidx"])), np.roll(pb, int(ib["splitidx"]))
        assert np.max(np.abs(wa - wb)) <= 1e-10 * wb.max()
        lo, hi = sorted((int(ia["splitidx"]), int(ib["splitidx"])))
        assert np.all(wb[lo:hi] < 1e-9 * wb.max())
