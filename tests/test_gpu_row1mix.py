"""The single-block kernel at sizes that are no power of two (2^a 3^b 5^c 7^d)
and with a block per dataset, against cuFFT's path of the same engine: every
radix first and last, odd half sizes, the smallest and largest sizes, batches
on either side of one block per SM, several datasets, rejected rows.
Tolerances as between the FFT forms elsewhere; the maps' noise keeps the
pixels inside the P(D)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ndata,nprop,binned", [
    (256, 1, 3, True), (294, 1, 3, True), (486, 1, 4, True), (512, 2, 5, True),
    (1000, 1, 148, True), (1000, 1, 149, True), (2058, 3, 6, True), (3000, 2, 74, True),
    (3000, 2, 75, True), (4096, 3, 7, True), (4096, 2, 80, True), (5000, 1, 5, False),
    (6000, 3, 9, False), (7056, 1, 4, True), (8100, 1, 3, True), (8192, 4, 5, True)])
def test_mixed_sizes_and_block_per_dataset(gpu_ctx, n, ndata, nprop, binned):
    from pofd_affine_b200 import beam, calcLike, synth
    from pofd_affine_b200._lib import PofdError
    rng = np.random.default_rng(n + ndata)
    kp, kv = synth.knot_model(5, 0.002, 0.2, rng=rng)
    bm = synth.gaussian_beam(3.0)
    L = calcLike(gpu_ctx, kp, n, 700, binned, 300)
    L.addBeamSet(beam(bm, 6.0, True, 100))
    for d in range(ndata):
        s = 0.003 * (1 + 0.3 * d)
        L.addDataset(0, synth.make_map((40, 44 + d), 6.0, bm, kp, kv, 0.001, rng), s)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    L.setRRanges(th0)
    th = synth.proposals(th0, nprop, 0.02, rng=rng)
    th[0, -1] = 1.1
    th[1, 0] = np.nan
    th[2, -1] = -0.5
    out = []
    for mode in (0, 1):
        L.setFFT(mode)
        ll, st = L.getLogLikeBatch(th)
        pd = []
        for d in range(ndata):
            try:
                pd.append(L.getPD(0, d, th[0], setLog=False))
            except PofdError as e:
                pd.append(e.code)
        out.append((ll, st, pd))
    (l0, s0, p0), (l1, s1, p1) = out
    assert list(s0) == list(s1)
    ok = s1 == 0
    assert np.array_equal(np.isnan(l0), np.isnan(l1))
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
