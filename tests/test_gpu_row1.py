"""The single-block kernel of small 1D grids (n = 1024 ... 8192) against the
multi-kernel cuFFT path of the same engine, where its tiles, sides, cut-offs
and batch shapes can go wrong: both beam sides, node counts off the block
size, datasets of different noise, several beam sets, rejected rows, batches
on either side of its launch rules; and on fresh engines call after call.
Tolerances as between the FFT forms elsewhere: log-likelihood within 1e-7,
P(D) within 1e-10 of its peak, status codes equal, splits equal or together
at the bottom of the P(D) (below 1e-9 of the peak)."""
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


def _pd(L, bs, ds, th):
    """The P(D), or its error code where the model is one without."""
    from pofd_affine_b200._lib import PofdError
    try:
        return L.getPD(bs, ds, th, setLog=False)
    except PofdError as e:
        return e.code


@pytest.mark.parametrize("n,ni,neg,sigmas,nsets,nprop,nbins", [
    (1024, 300, False, [0.004], 1, 5, 200),
    (2048, 2048, True, [0.0025], 1, 12, 1000),
    (4096, 1501, True, [0.002, 0.006], 1, 41, 500),
    (4096, 5, False, [0.0025], 1, 3, 1),
    (4096, 2048, False, [0.0025], 3, 60, 0),
    (8192, 4096, False, [0.0008, 0.003], 1, 4, 1000),
    (8192, 1024, True, [0.003], 2, 80, 300),
])
def test_single_block_matches_multi_kernel(gpu_ctx, n, ni, neg, sigmas, nsets, nprop, nbins):
    from pofd_affine_b200 import beam, calcLike, synth
    rng = np.random.default_rng(n + ni)
    kp, kv = synth.knot_model(7, 0.002, 0.4, rng=rng)
    L = calcLike(gpu_ctx, kp, n, ni, nbins > 0, max(nbins, 1))
    for b in range(nsets):
        bm = _ring(3.0 + b) if neg else synth.gaussian_beam(3.0 + b)
        L.addBeamSet(beam(bm, 6.0, True, 100))
        for s in sigmas:
            L.addDataset(b, synth.make_map((64, 72), 6.0, bm, kp, kv, s, rng), s)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    L.setRRanges(th0)
    th = synth.proposals(th0, nprop, 0.02, rng=rng)
    th[1, -1] = 1.15
    if nprop > 4:
        th[2, 1] = np.nan    # an invalid model
        th[3, -1] = -0.5     # a negative sigma multiplier
    res = []
    for mode in (0, 1):
        L.setFFT(mode)
        ll, st = L.getLogLikeBatch(th)
        pd = [_pd(L, nsets - 1, d, th[1]) for d in range(len(sigmas))]
        res.append((ll, st, pd))
        kernels = L.kernelsPerEval()
        assert kernels == (2 + (nsets > 1) if mode == 0 else 8)
    if n < 8192:  # the four-step FFT on and off again is the automatic choice
        L.setTuning(own_fft=1)
        L.setTuning(own_fft=0)
        assert L.kernelsPerEval() == 2 + (nsets > 1)
    (l1, s1, p1), (l0, s0, p0) = res
    assert list(s1) == list(s0)
    ok = s0 == 0
    assert np.array_equal(np.isnan(l1), np.isnan(l0))
    assert np.all(np.abs(l1[ok] - l0[ok]) < 1e-7)
    for a, b in zip(p1, p0):
        assert isinstance(a, int) == isinstance(b, int)
        if isinstance(a, int):
            assert a == b
        else:
            (pa, ia), (pb, ib) = a, b
            wa, wb = np.roll(pa, int(ia["splitidx"])), np.roll(pb, int(ib["splitidx"]))
            assert np.max(np.abs(wa - wb)) <= 1e-10 * wb.max()
            lo, hi = sorted((int(ia["splitidx"]), int(ib["splitidx"])))
            assert np.all(wb[lo:hi] < 1e-9 * wb.max())
            assert abs(ia["mn"] - ib["mn"]) <= 1e-12 * abs(ib["mn"])
            assert abs(ia["var_noi"] - ib["var_noi"]) <= 1e-12 * ib["var_noi"]


def test_fresh_engines_call_after_call(gpu_ctx):
    """Every call sets up its engine anew (new device memory, no captured
    graph) with another noise: each gives that noise's P(D)."""
    from pofd_affine_b200 import PDFactory, beam, synth
    kp, kv = synth.knot_model(6, 0.002, 0.4, rng=1)
    bm = beam(synth.gaussian_beam(3.0), 6.0, True, 120)
    f = PDFactory(gpu_ctx, 512)
    sig = [0.002 + 0.0005 * k for k in range(6)]
    ref = {}
    for k in range(60):
        f.initPD(4096, 0.0, 0.45, kp, kv, bm)
        s = sig[k % 6]
        r = f.getPD(s, setLog=False)
        assert np.all(np.isfinite(r.pd)) and abs(r.pd.sum() * r.dflux - 1.0) < 1e-3
        if s in ref:
            assert np.array_equal(ref[s], r.pd)
        ref[s] = r.pd
    assert len({float(p.max()) for p in ref.values()}) == 6
