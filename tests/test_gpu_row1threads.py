"""Engines of different sizes that share an instantiation of the single-block
kernel, each launching from a thread of its own: a launch's shared memory must
not be limited by what the other engine needs."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small,large", [((256, 64), (6000, 4096)), ((4096, 64), (4096, 4096))])
def test_engines_in_threads(gpu_ctx, small, large):
    from pofd_affine_b200 import Context, beam, calcLike, synth
    kp, kv = synth.knot_model(6, 0.002, 0.3, rng=1)
    bm = synth.gaussian_beam(3.0)
    th0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    th = synth.proposals(th0, 3, 0.01, rng=2)
    Ls, refs, errs = [], [], []
    for n, ni in (small, large):
        L = calcLike(Context(0), kp, n, ni, True, 300)
        L.addBeamSet(beam(bm, 6.0, True, 100))
        L.addDataset(0, synth.make_map((40, 40), 6.0, bm, kp, kv, 0.002, 3), 0.003)
        L.setRRanges(th0)
        Ls.append(L)
        refs.append(L.getLogLikeBatch(th))

    def work(L):
        try:
            L.profileStages(th, reps=4000)  # launches, a wait after each
        except Exception as e:
            errs.append(e)

    ts = [threading.Thread(target=work, args=(L,)) for L in Ls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs, errs
    for L, (ll, st) in zip(Ls, refs):
        assert np.all(st == 0) and np.array_equal(L.getLogLikeBatch(th)[0], ll)
