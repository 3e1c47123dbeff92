"""A P(D) factory hands its memory from one initPD to the next: sizes going up
and down, FFTs of all three kinds (one block, own, cuFFT), node counts and two
factories in turn give bit for bit what a factory of their own gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_reused_memory_gives_the_same_pd(gpu_ctx):
    from pofd_affine_b200 import PDFactory, beam, synth
    kp, kv = synth.knot_model(6, 0.002, 0.4, rng=1)
    bm = beam(synth.gaussian_beam(3.0), 6.0, True, 120)
    fs = {ni: PDFactory(gpu_ctx, ni) for ni in (512, 2048)}
    ref = {}
    seq = [(4096, 512), (1024, 2048), (65536, 512), (6000, 2048), (2048, 512), (16384, 2048),
           (4096, 2048), (1024, 512)]
    for rep in range(3):
        for n, ni in seq[rep:] + seq[:rep]:
            f = fs[ni]
            f.initPD(n, 0.0, 0.45, kp, kv, bm)
            r = f.getPD(0.0025, setLog=False)
            if (n, ni) not in ref:
                g = PDFactory(gpu_ctx, ni)
                g.initPD(n, 0.0, 0.45, kp, kv, bm)
                ref[n, ni] = (g.getPD(0.0025, setLog=False), g.getR())
            q, R = ref[n, ni]
            assert np.array_equal(q.pd, r.pd) and q.minflux == r.minflux and q.dflux == r.dflux
            assert np.array_equal(R, f.getR())
