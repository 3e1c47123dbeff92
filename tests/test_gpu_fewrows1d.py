"""The 1D inverse transform in one pass (spectra cut by the noise to a few
rows of 256 bins) and its reductions, against cuFFT's path of the same engine
at the edges of its rule: cut-offs on both sides of each row boundary and of
the limit of 8 rows, so that rows of both kinds meet in one batch and in one
beam set; every size of the own FFT; a dataset without noise.  Tolerances as
between the FFT forms elsewhere: log-likelihood within 1e-7, P(D) within
1e-10 of its peak (values between differing splits below 1e-9 of it).  The
maps' own noise is small, so that every pixel lies inside the P(D) of every
multiplier: pixels out where the P(D) is the transforms' rounding (1e-16 of
its peak) have logarithms that no two FFTs share."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EDGES = [180, 255, 256, 257, 300, 511, 512, 513, 767, 768, 769, 1022, 1023, 1024, 1025, 1300]


@pytest.mark.parametrize("n,sigmas", [(4096, [0.002]), (8192, [0.002, 0.003]), (16384, [0.002]),
                                      (32768, [0.0015, 0.004]), (65536, [0.002, 0.0021]),
                                      (131072, [0.002])])
def test_one_pass_inverse_matches_cufft(gpu_ctx, n, sigmas):
    from pofd_affine_b200 import beam, calcLike, synth
    from pofd_affine_b200._lib import PofdError
    rng = np.random.default_rng(n)
    kp, kv = synth.knot_model(6, 0.002, 0.4, rng=rng)
    bm = synth.gaussian_beam(3.0)
    L = calcLike(gpu_ctx, kp, n, 1500, True, 400)
    L.addBeamSet(beam(bm, 6.0, True, 100))
    for s in sigmas:
        L.addDataset(0, synth.make_map((60, 60), 6.0, bm, kp, kv, 0.0003, rng), s)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    L.setRRanges(th0)
    L.setFFT(0)
    L.setTuning(rfill_mode=1)  # the four-step sequence at every size
    _, info = L.getPD(0, 0, th0, setLog=False)
    # the multipliers that put the first dataset's cut-off
    # ceil(12 n dflux / (2 pi sigma)) + 1 at each edge
    mult = [12.0 * n * info["dflux"] / (2 * np.pi * sigmas[0] * (kc - 1.5)) for kc in EDGES]
    th = np.tile(th0, (len(EDGES), 1))
    th[:, -1] = mult
    out = []
    for mode in (0, 1):
        L.setFFT(mode)
        if mode == 0:
            L.setTuning(rfill_mode=1)
        ll, st = L.getLogLikeBatch(th)
        pd = []
        for k in range(len(EDGES)):
            try:
                pd.append(L.getPD(0, len(sigmas) - 1, th[k], setLog=False))
            except PofdError as e:
                pd.append(e.code)
        out.append((ll, st, pd))
        assert L.kernelsPerEval() == (10 if mode == 0 else 8)
    (l0, s0, p0), (l1, s1, p1) = out
    assert list(s0) == list(s1) and np.sum(s0 == 0) >= 8
    ok = s1 == 0
    assert np.all(np.abs(l0[ok] - l1[ok]) < 1e-7)
    for a, b in zip(p0, p1):
        assert isinstance(a, int) == isinstance(b, int)
        if isinstance(a, int):
            assert a == b
            continue
        (pa, ia), (pb, ib) = a, b
        wa, wb = np.roll(pa, int(ia["splitidx"])), np.roll(pb, int(ib["splitidx"]))
        assert np.max(np.abs(wa - wb)) <= 1e-10 * wb.max()
        lo, hi = sorted((int(ia["splitidx"]), int(ib["splitidx"])))
        assert np.all(wb[lo:hi] < 1e-9 * wb.max())
        assert abs(ia["mn"] - ib["mn"]) <= 1e-9 * abs(ib["mn"])


def test_one_pass_inverse_without_noise(gpu_ctx):
    """No noise or next to none leaves no cut: the general passes; codes and
    values as cuFFT's."""
    from pofd_affine_b200 import beam, calcLike, synth
    rng = np.random.default_rng(3)
    kp, kv = synth.knot_model(6, 0.002, 0.4, rng=rng)
    bm = synth.gaussian_beam(3.0)
    L = calcLike(gpu_ctx, kp, 16384, 1500, True, 400)
    L.addBeamSet(beam(bm, 6.0, True, 100))
    L.addDataset(0, synth.make_map((60, 60), 6.0, bm, kp, kv, 0.002, rng), 0.002)
    th = np.tile(np.concatenate([kv, [1.0]]).astype(np.float32), (4, 1))
    th[:, -1] = [1.0, 0.0, -1.0, 0.01]
    L.setRRanges(th[0])
    r = []
    for mode in (0, 1):
        L.setFFT(mode)
        r.append(L.getLogLikeBatch(th))
    assert list(r[0][1]) == list(r[1][1])
    fin = np.isfinite(r[1][0])
    assert np.array_equal(fin, np.isfinite(r[0][0]))
    assert np.all(np.abs(r[0][0][fin] - r[1][0][fin]) <= 1e-7 * np.maximum(1.0, np.abs(r[1][0][fin])))
