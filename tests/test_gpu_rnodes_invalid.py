"""R at the nodes of a model without one (an undefined knot value) is 0, not
what the device memory held before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_nodes_of_an_invalid_model(gpu_ctx):
    import torch
    from pofd_affine_b200 import beam, calcLike, synth
    kp, kv = synth.knot_model(6, 0.002, 0.3, rng=1)
    bm = synth.gaussian_beam(3.0)
    L = calcLike(gpu_ctx, kp, 1024, 8000, True, 100)
    L.addBeamSet(beam(bm, 6.0, True, 60))
    L.addDataset(0, synth.make_map((40, 40), 6.0, bm, kp, kv, 0.002, 3), 0.003)
    th = np.concatenate([kv, [1.0]]).astype(np.float32)
    L.setRRanges(th)
    assert np.any(L.getRNodes(0, th, 8000)[1] > 0)
    bad = th.copy()
    bad[2] = np.nan
    for _ in range(5):
        junk = [torch.full((1 << 18,), 7.0, dtype=torch.float64, device="cuda") for _ in range(8)]
        torch.cuda.synchronize()
        del junk
        torch.cuda.empty_cache()
        x, R = L.getRNodes(0, bad, 8000)
        assert np.all(np.diff(x) > 0) and np.all(R == 0.0)
