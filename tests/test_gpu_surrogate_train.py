"""The surrogate's training kernels where their tiles can go wrong: hidden
widths off the 128-row tile, row counts off it, one row, and row counts that
give each tile width (16 ... 128 columns).  Gradients and loss against the CPU
oracle with the tolerances of the main gradient test (bf16 activations), the
forward pass against itself in narrow tiles; one training step against Adam's first step, which is -lr
sign(g) to eps / |g| and the rounding of the weights (1e-7 / lr), wherever the
oracle's gradient is well away from zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NAMES = ["W1", "b1", "W2", "b2", "W3", "b3", "w4", "b4"]


def _pairs(n, k, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, k))
    ll = -0.5 * (x * x).sum(1) - 0.1 * np.sin(2.0 * x).sum(1) - 100.0
    th = x @ (np.eye(k) + 0.1 * rng.normal(size=(k, k))).T - 2.0
    return np.concatenate([th, np.ones((n, 1))], 1).astype(np.float32), ll


def _oracle(S, th, ll, k, H):
    import mlp_oracle
    sc = S.scaling()
    params = [p.astype(np.float64) for p in S.getParams()]
    x = mlp_oracle.standardise(th, list(range(k)), sc["mu"], sc["W"])
    t = (np.maximum(ll - sc["ymax"], -sc["clip"]) / sc["ys"]).astype(np.float32).astype(np.float64)
    return sc, params, x, mlp_oracle.gradients(params, H, x, t)


@pytest.mark.parametrize("k,H,n", [(1, 16, 2), (3, 112, 129), (16, 144, 700), (5, 512, 1300),
                                   (4, 512, 2500), (6, 512, 5000)])
def test_gradients_at_tile_edges(gpu_ctx, k, H, n):
    import mlp_oracle
    from pofd_affine_b200.surrogate import Surrogate
    th, ll = _pairs(n, k, k + H + n)
    S = Surrogate(gpu_ctx, k + 1, list(range(k)), hidden=H, capacity=8192, seed=3)
    S.addPairs(th, ll)
    g, loss = S.gradients(n)
    sc, params, x, (og, oloss) = _oracle(S, th, ll, k, H)
    assert abs(loss - oloss) <= 1e-3 * oloss
    for name, a, b in zip(NAMES, g, og):
        rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
        assert rel < 2e-2, (name, rel)
    # forward in its tile width against the narrow tiles of 100-row calls:
    # only the order of the H products of an output differs, two FP32 sums
    # each within H 2^-24 sum |h3 w4| of the exact one
    _, acts = mlp_oracle.forward(params, H, x)
    bound = 2 * H * 2.0 ** -24 * (np.abs(acts[-1]) @ np.abs(params[6])) * sc["ys"]
    parts = np.concatenate([S.predict(th[i:i + 100]) for i in range(0, n, 100)])
    assert np.all(np.abs(S.predict(th) - parts) <= bound + 1e-12)


def _picked(it, seed, slots, n):
    """Rows of a minibatch: splitmix64's finaliser of (iteration, slot)."""
    M = (1 << 64) - 1
    rows = []
    for r in range(slots):
        v = seed ^ ((it * 0x9E3779B97F4A7C15) & M) ^ ((r * 0xBF58476D1CE4E5B9) & M)
        v = ((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & M
        v = ((v ^ (v >> 27)) * 0x94D049BB133111EB) & M
        v ^= v >> 31
        rows.append(((v >> 32) * n) >> 32)
    return np.array(rows)


@pytest.mark.parametrize("k,H,n,batch", [(2, 16, 300, 1), (14, 256, 2000, 512), (5, 144, 1000, 300)])
def test_first_step_is_adams(gpu_ctx, k, H, n, batch):
    from pofd_affine_b200.surrogate import Surrogate
    th, ll = _pairs(n, k, 7)
    S = Surrogate(gpu_ctx, k + 1, list(range(k)), hidden=H, capacity=4096, seed=9)
    S.addPairs(th, ll)
    S.gradients(n)  # fixes the scaling
    rows = _picked(1, 9, batch, n)
    _, params, _, (og, _) = _oracle(S, th[rows], ll[rows], k, H)
    lr = 1e-3
    S.train(1, batch=batch, lr=lr)
    for name, p0, p1, g in zip(NAMES, params, S.getParams(), og):
        g = np.asarray(g, np.float64).ravel()
        big = np.abs(g) > 0.2 * np.abs(g).max()
        step = (p1.astype(np.float64) - p0).ravel()[big]
        assert np.max(np.abs(step + lr * np.sign(g[big]))) < 1e-2 * lr, name


@pytest.mark.parametrize("k,n,far,same", [(1, 2, 0, False), (16, 65, 0, False), (3, 160, 120, False),
                                          (5, 149, 0, True), (14, 8001, 3000, False),
                                          (7, 70000, 0, False)])
def test_scaling_matches_float64(gpu_ctx, k, n, far, same):
    """Mean, whitening and target scaling against numpy in 64 bits: few and
    many pairs (blocks of one row and of several hundred), most of them far
    below the maximum (too few near it: all are used), two equal inputs (no
    Cholesky factor: diagonal scaling).  The mean and W are stored in FP32
    (6e-8); the sums differ by their order only, and W by that times the
    covariance's condition (< 1e3 here)."""
    from pofd_affine_b200.surrogate import Surrogate
    th, ll = _pairs(n, k, 11)
    th[:, :k] += 5.0
    if same:
        th[:, 1] = th[:, 0]
    ll[:far] -= 500.0
    S = Surrogate(gpu_ctx, k + 1, list(range(k)), hidden=16, capacity=max(n, 128), seed=1)
    S.addPairs(th, ll)
    S.gradients(2)
    sc = S.scaling()
    clip = 25.0 + 2.5 * k
    d = np.maximum(ll - ll.max(), -clip)
    assert sc["ymax"] == ll.max() and sc["clip"] == clip
    assert abs(sc["ys"] - d.std()) <= 1e-12 * d.std()
    use = ll - ll.max() > -clip
    if use.sum() < max(2 * k, 64):
        use[:] = True
    x = th[use, :k].astype(np.float64)
    assert np.max(np.abs(sc["mu"][:k] - x.mean(0)) / np.abs(x.mean(0))) < 1e-7
    cov = np.cov(x.T, bias=True).reshape(k, k)
    W = np.zeros((16, 16))
    W[:k, :k] = np.diag(1 / np.sqrt(np.diag(cov))) if same else np.linalg.inv(np.linalg.cholesky(cov))
    assert sc["whitened"] == (not same)
    assert np.max(np.abs(sc["W"] - W)) < 1e-7 * np.abs(W).max()
