"""A P(D) factory set up again and again holds the memory of two set-ups at
most, whether or not a P(D) is asked of it: sizes that grow slowly, so that no
block of one set-up is large enough for the next, with R only, with set-ups
alone, and with P(D)s that fail."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use", ["R", "nothing", "failing P(D)"])
def test_memory_is_bounded(gpu_ctx, use):
    import torch
    from pofd_affine_b200 import PDFactory, beam, synth
    from pofd_affine_b200._lib import PofdError
    kp, kv = synth.knot_model(6, 0.002, 0.4, rng=1)
    bm = beam(synth.gaussian_beam(3.0), 6.0, True, 120)
    f = PDFactory(gpu_ctx, 512)
    free = []
    for k in range(40):
        f.initPD(400000 + 3000 * k, 0.0, 0.45, kp, kv, bm)
        if use == "R":
            f.getR()
        elif use != "nothing":
            with pytest.raises(PofdError):
                f.getPD(50.0)  # no split point within such a noise
        free.append(torch.cuda.mem_get_info()[0])
    one = 30 << 20  # more than one set-up of 517000 points takes (20 MB of rows, tables)
    assert free[3] - min(free[4:]) < 2 * one, [(free[3] - x) >> 20 for x in free]
