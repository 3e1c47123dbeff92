"""Which path a batch takes, by the launches of its evaluation: the single-block
kernel is two (three with several beam sets), the kernels around cuFFT eight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(ctx, n, ndata, nsets=1, npix=0):
    from pofd_affine_b200 import beam, calcLike, synth
    kp, kv = synth.knot_model(5, 0.002, 0.2, rng=n)
    bm = synth.gaussian_beam(3.0)
    m = synth.make_map((64, 64), 6.0, bm, kp, kv, 0.001, 1).ravel()
    L = calcLike(ctx, kp, n, 200, npix == 0, 100)
    for b in range(nsets):
        L.addBeamSet(beam(bm, 6.0, True, 50))
        for d in range(ndata):
            L.addDataset(b, np.resize(m, npix) if npix else m, 0.003 + 0.0001 * d)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    L.setRRanges(th0)
    return L, th0


def _launches(L, th0, rows):
    ll, st = L.getLogLikeBatch(np.tile(th0, (rows, 1)))
    assert np.all(st == 0) and np.all(np.abs(ll - ll[0]) < 1e-7)
    return L.kernelsPerEval()


def test_mixed_size_counts_by_batch(gpu_ctx):
    L, th0 = _engine(gpu_ctx, 1000, 1)
    assert L.kernelsPerEval() == 2  # one row
    assert _launches(L, th0, 200) == 8
    assert _launches(L, th0, 100) == 2


@pytest.mark.parametrize("n,ndata,npix,rows,launches", [
    (1024, 64, 0, 2, 2), (1024, 64, 0, 3, 8), (2048, 8, 0, 18, 2), (2048, 8, 0, 20, 8),
    (4096, 2, 0, 80, 2), (4096, 40, 0, 20, 8), (8192, 40, 0, 20, 10), (1024, 1, 0, 600, 2),
    (1024, 1, 60000, 148, 2), (1024, 1, 60000, 300, 8), (1024, 2, 30000, 300, 8),
    (7290, 1, 0, 1, 2), (7500, 2, 0, 3, 8), (8100, 1, 0, 1, 8), (8100, 1, 0, 31, 8),
    (8100, 1, 0, 32, 2), (8100, 4, 0, 37, 2), (8100, 4, 0, 38, 8)])
def test_serial_work_of_a_block(gpu_ctx, n, ndata, npix, rows, launches):
    """A block takes the datasets of its row, and their bins, in turn: many of
    them go to the separate kernels unless each has a block of its own.  So do
    the largest mixed sizes in the smallest batches."""
    L, th0 = _engine(gpu_ctx, n, ndata, 1, npix)
    assert _launches(L, th0, rows) == launches
    ll = L.getLogLikeBatch(np.tile(th0, (rows, 1)))[0]
    L.setFFT(1)
    assert np.all(np.abs(L.getLogLikeBatch(np.tile(th0, (rows, 1)))[0] - ll) < 1e-7 * (1 + npix * ndata / 4096))
