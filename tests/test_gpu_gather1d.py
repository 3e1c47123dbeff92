"""The pixels' part of the 1D likelihood at pixel counts on either side of the
groups that a thread takes together, in the kernels that hold it: one block per
row with 512 and 256 threads, and the finishing kernel behind cuFFT and behind
the four-step FFT.  Reference: the P(D) that the engine returns, interpolated in
float64; both sides round some thousand terms of size ten, so 1e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 544, 767, 769, 1023, 1024, 1025, 1055, 1537,
          2047, 2049, 2560, 4097]


@pytest.mark.parametrize("n,mode,rows", [(1024, 0, 1), (1024, 0, 200), (1024, 1, 2), (16384, 0, 2)])
def test_pixel_counts(gpu_ctx, n, mode, rows):
    from pofd_affine_b200 import beam, calcLike, synth
    rng = np.random.default_rng(n + rows)
    kp, kv = synth.knot_model(5, 0.002, 0.2, rng=rng)
    bm = beam(synth.gaussian_beam(3.0), 6.0, True, 60)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    sigma = 0.003
    wide = calcLike(gpu_ctx, kp, n, 300, False, 10)  # R range of all the counts
    wide.addBeamSet(bm)
    wide.addDataset(0, rng.normal(0.0, 0.004, 64), sigma)
    wide.setRRanges(th0)
    span = abs(wide.getPD(0, 0, th0)[1]["pd_minflux"])
    for count in COUNTS:
        px = rng.normal(0.0, 0.3 * span, count)
        px[:: 37] = -3.0 * span  # below the grid
        L = calcLike(gpu_ctx, kp, n, 300, False, 10)
        L.addBeamSet(bm)
        L.addDataset(0, px, sigma, meansub=False)
        L.setRRanges(th0)
        L.setFFT(mode)
        ll, st = L.getLogLikeBatch(np.tile(th0, (rows, 1)))
        assert np.all(st == 0) and np.all(ll == ll[0])
        lp, info = L.getPD(0, 0, th0, setLog=True)
        x = (px - info["pd_minflux"]) / info["dflux"]
        i = np.clip(x.astype(np.int64), 0, n - 2)
        t = x - i
        v = np.where(x <= 0, lp[0], np.where(x >= n - 2, lp[n - 1],
                                             (1.0 - t) * lp[i] + t * lp[i + 1]))
        want = np.log(2.0) * v.sum() + 0.5 * count * (np.log(2 * np.pi * sigma ** 2) + 1.0)
        assert abs(ll[0] - want) < 1e-8, (count, ll[0], want)
