"""Colour curves at their limits: an infinite offset is a Gaussian that is 0
everywhere, so the model is one without sources (the likelihood of an offset
far outside every flux ratio); a sigma of 0 or an undefined offset stays an
error, and neither touches the rows beside it."""
import numpy as np
import pytest

from test_gpu_2d import build2, spec2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,edge", [(256, True), (512, True), (512, False)])
def test_infinite_offset(orc, gpu_ctx, n, edge):
    s = spec2(n=n, nedge=48, edge=edge, nsig=1, noff=1, shape=(48, 48))
    G = build2(orc, gpu_ctx, s)[1]
    K = len(s["kp"])
    th = np.tile(s["th"], (7, 1))
    th[1, K + 1] = np.inf
    th[2, K + 1] = -np.inf
    th[3, K + 1] = 300.0   # exp(-(300 / 0.2)^2 / 2) = 0
    th[4, K + 1] = -300.0
    th[5, K] = 0.0
    th[6, K + 1] = np.nan
    ll, st = G.getLogLikeBatch(th)
    assert np.all(st[:5] == 0) and np.all(st[5:] != 0)
    assert np.all(np.isfinite(ll[:5])) and np.all(np.isnan(ll[5:]))
    assert np.all(np.abs(ll[1:5] - ll[3]) <= 1e-12 * abs(ll[3]))
    assert ll[0] == G.getLogLikeBatch(np.tile(s["th"], (7, 1)))[0][0] != ll[3]
