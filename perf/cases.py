"""Performance cases of the P(D) likelihood library.

Each case is one piece of work that a fit with this library does through its
Python interface, on synthetic maps of the shapes, beams and noise levels of
the library's own configurations (pofd_affine_b200/synth.py):

  like1   calcLike.getLogLike / getLogLikeBatch: 1D log-likelihoods
  pd1     PDFactory.initPD + getPD: one 1D P(D)
  like2   calcLikeDouble.getLogLikeBatch: two-band log-likelihoods
  fields  likeSum of two two-band fields on device arrays
  chain   affineEnsemble.doSteps over a 1D likelihood, and the chain
  train   Surrogate.train and predict

listed() gives the fixed cases, draw() further ones of the same ranges,
prepare() builds what a program has in hand before the call, run() is one
call, work() counts the arithmetic and the bytes that the call cannot do
without, and exact() restates the likelihoods and the P(D) in plain float64
numpy / torch (natural splines by the Thomas algorithm, torch.fft), from the
same inputs.
"""
import ctypes
import math

import numpy as np
import torch

from pofd_affine_b200 import Context, PDFactory, beam, calcLike, calcLikeDouble, doublebeam, synth

DEV = "cuda" if torch.cuda.is_available() else "cpu"
PIX = 6.0            # arcsec, the pixel size of every configuration
NZEROPAD = 7.5       # noise sigmas of padding in the R range
SMALLLOG = -30.0     # log2 of a vanishing P(D)
HISTPAD = 0.0014419741739063218  # log2(1.001), padding of beam histograms

_context = None


def _ctx():
    global _context
    if _context is None:
        _context = Context(0)
    return _context


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one parameter vector at a time on the small 1D fit (6 knots, a
        # 256 x 256 map, n = 4096): what an optimiser or a script calls
        _like1("1d one", n=4096, nprop=1, knots=6, sets=1, data=1, side=256),
        # a half-ensemble of that fit (40 walkers), one sampler half-step
        _like1("1d half-ensemble", n=4096, nprop=20, knots=6, sets=1, data=1, side=256),
        # the batched fit: 10 knots, three beams, one map each, n = 65536,
        # 128 walkers' proposals
        _like1("1d batched", n=65536, nprop=128, knots=10, sets=3, data=1, side=500, hist=150),
        # the class's default FFT size, two maps per beam, an uneven batch
        _like1("1d default size", n=131072, nprop=33, knots=8, sets=2, data=2, side=200),
        # a size that is no power of two, a beam with negative lobes that is
        # not histogrammed away, pixels unbinned
        _like1("1d odd unbinned", n=6000, ninterp=1500, nprop=25, knots=7, sets=1, data=3,
               side=60, neg=True, binned=False),
        # one P(D) from explicit flux limits, as a model check or plot wants
        {"name": "1d P(D)", "kind": "pd1", "n": 4096, "ninterp": 2048, "knots": 6, "hist": 120,
         "neg": False, "noise": 0.0025},
        # the two-band fit: 8 knots, 3 sigma and 3 offset knots, n = 2048,
        # 64 walkers' proposals
        _like2("2d plain", n=2048, nprop=64, nedge=256, side=600, nbins=500),
        # the class's default FFT size and bins, a few proposals
        _like2("2d default size", n=4096, nprop=6, nedge=256, side=400, nbins=1000),
        # small two-band batch on a size that is no power of two, both maps'
        # beams with negative lobes, two datasets of the same beams
        _like2("2d odd", n=600, nprop=9, nedge=96, side=120, nbins=200, data=2, neg=True,
               hist=30),
        # the surviving proposals of a delayed-acceptance half-step on the
        # joint fit of two fields (n = 2048 and 1024), device arrays
        {"name": "2d two fields", "kind": "fields", "n": 2048, "n2": 1024, "nprop": 6,
         "nedge": 256, "side": 300, "nbins": 500},
        # sampler steps of the small 1D fit, 40 walkers, chain read back
        {"name": "1d chain", "kind": "chain", "n": 4096, "walkers": 40, "steps": 20,
         "knots": 6, "side": 256},
        # online training of the delayed-acceptance surrogate on the exact
        # pairs of a burn-in, then a half-ensemble's screening
        {"name": "surrogate", "kind": "train", "pairs": 8000, "inputs": 14, "hidden": 256,
         "iters": 20, "batch": 512, "rows": 64},
    ]


def _like1(name, n, nprop, knots, sets, data, side, ninterp=2048, hist=120, nbins=1000,
           neg=False, binned=True):
    return {"name": name, "kind": "like1", "n": n, "ninterp": ninterp, "nprop": nprop,
            "knots": knots, "sets": sets, "data": data, "side": side, "hist": hist,
            "nbins": nbins, "neg": neg, "binned": binned}


def _like2(name, n, nprop, nedge, side, nbins, data=1, neg=False, hist=100):
    return {"name": name, "kind": "like2", "n": n, "nprop": nprop, "nedge": nedge, "side": side,
            "nbins": nbins, "data": data, "neg": neg, "hist": hist, "nsigma": 3, "noffset": 3}


def draw(rng):
    """Another case of the listed ranges: FFT sizes both powers of two and
    not, batches spread over their logarithm."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["like1"] * 4 + ["like2"] * 4 + ["fields", "pd1", "chain", "train"])
    if kind == "like1":
        n = 1 << rng.randint(11, 17) if rng.random() < 0.7 else logint(2000, 40000)
        sets, data = rng.randint(1, 3), rng.randint(1, 2)
        nprop = logint(1, max(1, min(160, 65536 * 384 // (n * sets * data))))
        neg = rng.random() < 0.25
        c = _like1("", n, nprop, rng.randint(5, 12), sets, data, rng.randint(60, 300),
                   rng.choice([1024, 1500, 2048]), rng.choice([100, 120, 150]),
                   rng.choice([500, 1000]), neg, rng.random() < 0.85)
        if not c["binned"]:
            c["side"] = rng.randint(60, 90)
    elif kind == "like2":
        n = 1 << rng.randint(8, 12) if rng.random() < 0.75 else rng.randint(240, 900)
        neg = n <= 512 and rng.random() < 0.4
        cap = 2048 * 2048 * 64 // (n * n) // (4 if neg else 1)
        c = _like2("", n, logint(1, max(1, min(64, cap // 2))), min(rng.choice([64, 128, 256]), n),
                   rng.randint(100, 400), rng.choice([100, 200, 500]), 1, neg,
                   30 if neg else 100)
        c["data"] = 2 if rng.random() < 0.25 else 1
        c["nsigma"], c["noffset"] = rng.choice([(1, 1), (2, 2), (3, 3), (4, 3)])
    elif kind == "fields":
        n = rng.choice([512, 1024, 2048])
        c = {"kind": "fields", "n": n, "n2": n // 2, "nprop": logint(1, 64),
             "nedge": rng.choice([64, 128, 256]), "side": rng.randint(100, 300),
             "nbins": rng.choice([200, 500])}
    elif kind == "pd1":
        c = {"kind": "pd1", "n": rng.choice([2048, 3000, 4096, logint(2048, 6000)]),
             "ninterp": rng.choice([1024, 2048]), "knots": rng.randint(5, 8),
             "hist": rng.choice([0, 100, 120]), "neg": rng.random() < 0.3,
             "noise": rng.uniform(0.002, 0.004)}
    elif kind == "chain":
        c = {"kind": "chain", "n": rng.choice([4096, 8192, 16384]),
             "walkers": 2 * rng.randint(10, 64), "steps": rng.randint(5, 30),
             "knots": rng.randint(5, 8), "side": rng.randint(64, 256)}
    else:
        c = {"kind": "train", "pairs": rng.randint(2000, 20000), "inputs": rng.randint(6, 14),
             "hidden": rng.choice([128, 256, 384]), "iters": rng.randint(5, 30),
             "batch": rng.choice([256, 512, 1024]), "rows": rng.randint(8, 128)}
    c.pop("name", None)
    return c


# ----------------------------------------------------------------- inputs
def _ring(fwhm, nfwhm, depth):
    """A Gaussian beam with a shallow negative ring, the shape a matched
    filter gives a beam."""
    g = synth.gaussian_beam(fwhm, nfwhm)
    y, x = np.mgrid[0:g.shape[0], 0:g.shape[1]]
    c = g.shape[0] // 2
    r2 = ((x - c) ** 2 + (y - c) ** 2) / (2.0 * fwhm) ** 2
    b = g - depth * r2 * np.exp(1.0 - r2)
    return b / b.max()


def _inputs1(c, seed):
    """Beams, maps, knots and parameter rows of a 1D fit."""
    rng = np.random.default_rng(seed)
    kp, kv = synth.knot_model(c["knots"], 0.001 if c["knots"] > 8 else 0.002,
                              0.800 if c["knots"] > 8 else 0.400, rng=rng)
    fwhm, noise = [3.0, 4.2, 6.0], [0.0020, 0.0031, 0.0050]
    beams, maps, sig = [], [], []
    for b in range(c["sets"]):
        bm = _ring(fwhm[b], 9.0, 0.05) if c["neg"] else synth.gaussian_beam(fwhm[b])
        beams.append(bm)
        s = [noise[b] * (1.0 + 0.4 * d) for d in range(c["data"])]
        sig.append(s)
        maps.append([synth.make_map((c["side"], c["side"] + 7 * d), PIX, bm, kp, kv, s[d], rng)
                     for d in range(c["data"])])
    theta0 = np.concatenate([kv, [1.0]]).astype(np.float32)
    theta = synth.proposals(theta0, c["nprop"], 0.02, rng=rng)
    return {"kp": kp, "beams": beams, "maps": maps, "sig": sig, "theta0": theta0,
            "theta": theta}


def _build1(c, q):
    L = calcLike(_ctx(), q["kp"], c["n"], c["ninterp"], c["binned"], c["nbins"])
    for b, bm in enumerate(q["beams"]):
        L.addBeamSet(beam(bm, PIX, c["hist"] > 0, c["hist"], 1e-5))
        for m, s in zip(q["maps"][b], q["sig"][b]):
            L.addDataset(b, m, s)
    L.setRRanges(q["theta0"])
    return L


def _chain1(c):
    return dict(_like1("", c["n"], c["walkers"], c["knots"], 1, 1, c["side"]))


def _inputs_pd1(c, seed):
    rng = np.random.default_rng(seed)
    kp, kv = synth.knot_model(c["knots"], 0.002, 0.400, rng=rng)
    bm = _ring(3.0, 9.0, 0.05) if c["neg"] else synth.gaussian_beam(3.0)
    noise = c["noise"] * rng.uniform(0.9, 1.1)
    return {"kp": kp, "kv": kv, "bm": bm, "noise": noise,
            "lo": -kp[-1] * 1.05 * max(0.0, -float(bm.min())),
            "hi": 1.05 * kp[-1] * float(bm.max()) + NZEROPAD * noise}


def _inputs2(c, seed, fields=1):
    """Beams, map pairs, knots and parameter rows of a two-band fit."""
    rng = np.random.default_rng(seed)
    ns, no = c.get("nsigma", 3), c.get("noffset", 3)
    kp, kv = synth.knot_model(8, 0.002, 0.500, rng=rng)
    sk = np.logspace(math.log10(0.002), math.log10(0.5), ns)
    sv = np.linspace(0.15, 0.3, ns).astype(np.float32)
    ok = np.logspace(math.log10(0.002), math.log10(0.5), no)
    ov = (math.log(0.7) + rng.normal(0, 0.02, no)).astype(np.float32)
    if c.get("neg"):
        b1, b2 = _ring(3.0, 7.0, 0.04), _ring(4.2, 5.0, 0.04)
    else:
        b1, b2 = synth.gaussian_beam(3.0, nfwhm=39 / 3.0), synth.gaussian_beam(4.2)
    sfn = lambda f: np.interp(f, sk, sv)  # noqa: E731
    ofn = lambda f: np.interp(f, ok, ov)  # noqa: E731
    sig = (0.0025, 0.0028)
    nmaps = c.get("data", 1)
    maps = [[synth.make_map_pair((c["side"], c["side"] + 5 * d), PIX, b1, b2, kp, kv, sfn, ofn,
                                 sig[0], sig[1], rng) for d in range(nmaps)]
            for _ in range(fields)]
    theta0 = np.concatenate([kv, sv, ov, [1.0, 1.0]]).astype(np.float32)
    theta = synth.proposals(theta0, c["nprop"], 0.01, rng=rng)
    theta[:, -2:] = 1.0
    return {"kp": kp, "sk": sk, "ok": ok, "b1": b1, "b2": b2, "maps": maps, "sig": sig,
            "theta0": theta0, "theta": theta}


def _build2(c, q, n, nedge, field):
    L = calcLikeDouble(_ctx(), q["kp"], q["sk"], q["ok"], n, nedge, True, c["nbins"])
    L.addBeamSet(doublebeam(q["b1"], q["b2"], PIX, True, c.get("hist", 100), 1e-6))
    for m1, m2 in q["maps"][field]:
        L.addDataset(0, m1, m2, *q["sig"])
    L.setRRanges(q["theta0"])
    return L


# ------------------------------------------------------------ prepare, run
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "like1":
        q = _inputs1(c, seed)
        L = _build1(c, q)
        L.reserve(c["nprop"])
        return {"kind": kind, "L": L, "theta": q["theta"], "one": c["nprop"] == 1}
    if kind == "pd1":
        q = _inputs_pd1(c, seed)
        q["beam"] = beam(q["bm"], PIX, c["hist"] > 0, c["hist"], 1e-5)
        return {"kind": kind, "f": PDFactory(_ctx(), c["ninterp"]), "n": c["n"], **q}
    if kind == "like2":
        q = _inputs2(c, seed)
        L = _build2(c, q, c["n"], c["nedge"], 0)
        L.reserve(c["nprop"])
        return {"kind": kind, "L": L, "theta": q["theta"]}
    if kind == "fields":
        from pofd_affine_b200.mcmc import likeSum
        q = _inputs2(c, seed, 2)
        La = _build2(c, q, c["n"], c["nedge"], 0)
        Lb = _build2(c, q, c["n2"], c["nedge"] // 2, 1)
        for L in (La, Lb):
            L.reserve(c["nprop"])
        return {"kind": kind, "S": likeSum(_ctx(), [La, Lb]),
                "theta": torch.from_numpy(q["theta"]).cuda(),
                "logl": torch.empty(c["nprop"], dtype=torch.float64, device="cuda"),
                "status": torch.empty(c["nprop"], dtype=torch.int32, device="cuda")}
    if kind == "chain":
        from pofd_affine_b200.mcmc import affineEnsemble
        k = _chain1(c)
        q = _inputs1(k, seed)
        L = _build1(k, q)
        E = affineEnsemble(_ctx(), L, c["walkers"], c["knots"] + 1, seed=seed)
        E.setParamFixed(c["knots"])
        for p in range(c["knots"]):
            E.setParamLimits(p, float(q["theta0"][p]) - 0.5, float(q["theta0"][p]) + 0.5)
        E.setErrorPolicy(True)  # a step whose P(D) cannot be unwrapped is rejected
        return {"kind": kind, "E": E, "walkers": q["theta"], "steps": c["steps"]}
    if kind == "train":
        from pofd_affine_b200.surrogate import Surrogate
        rng = np.random.default_rng(seed)
        k = c["inputs"]
        # pairs of a burn-in: correlated parameters, a curved log-likelihood
        A = rng.normal(size=(k, k)) * 0.02 + 0.05 * np.eye(k)
        x = rng.normal(size=(c["pairs"], k))
        ll = -0.5 * (x * x).sum(1) - 0.1 * np.sin(2.0 * x).sum(1) - 1.5e5
        th = np.concatenate([x @ A.T - 2.0, np.ones((c["pairs"], 1))], 1).astype(np.float32)
        S = Surrogate(_ctx(), k + 1, list(range(k)), hidden=c["hidden"], capacity=c["pairs"],
                      seed=seed % 1000 + 1)
        S.addPairs(th, ll)
        return {"kind": kind, "S": S, "w0": S.getParams(), "iters": c["iters"],
                "batch": c["batch"], "rows": th[:c["rows"]]}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "like1":
        if state["one"]:
            ll, invalid = state["L"].getLogLike(state["theta"][0])
            return np.float64(ll), invalid
        return state["L"].getLogLikeBatch(state["theta"])
    if kind == "pd1":
        f = state["f"]
        f.initPD(state["n"], state["lo"], state["hi"], state["kp"], state["kv"], state["beam"])
        r = f.getPD(state["noise"], setLog=False)
        return {"pd": r.pd, "minflux": np.float64(r.minflux), "dflux": np.float64(r.dflux)}
    if kind == "like2":
        return state["L"].getLogLikeBatch(state["theta"])
    if kind == "fields":
        from pofd_affine_b200._lib import check, lib
        th = state["theta"]
        check(lib().pofd_likesum_eval_batch_device(
            state["S"].h, th.shape[0], ctypes.c_void_p(th.data_ptr()), th.shape[1],
            ctypes.c_void_p(state["logl"].data_ptr()),
            ctypes.c_void_p(state["status"].data_ptr()), None))
        return state["logl"], state["status"]
    if kind == "chain":
        E = state["E"]
        E.initChains(state["walkers"])
        E.clearChain()
        E.doSteps(state["steps"])
        return E.getChain()
    S = state["S"]
    S.setParams(state["w0"])
    loss = S.train(state["iters"], state["batch"])
    return {"loss": loss, "weights": S.getParams(), "logl": S.predict(state["rows"])}


# ------------------------------------------------------------------- work
# Flops counted per unit: 25 for a term of the R sums (a spline or a
# quadratic, a 2^x, a multiply-add), 15 for a point of the 1D R grid, 40 for
# a spectrum bin (exp, sin, cos, products), 6 for a point of the P(D) scan.
def work(case):
    c, kind = case, case["kind"]
    if kind == "like1":
        f = _flops1(c, _inputs1(dict(c, nprop=1, side=64, data=1), 0), c["nprop"], c["data"])
        pix = c["nbins"] * 12 if c["binned"] else c["side"] * c["side"] * 8
        return {"flops": f, "bytes": c["nprop"] * (4 * c["knots"] + 16) + c["sets"] * c["data"] * pix}
    if kind == "pd1":
        q = _inputs_pd1(c, 0)
        k = {"n": c["n"], "ninterp": c["ninterp"], "hist": c["hist"]}
        return {"flops": _flops1(k, {"kp": q["kp"], "beams": [q["bm"]]}, 1, 1),
                "bytes": 8.0 * c["n"]}
    if kind == "like2":
        return {"flops": c["nprop"] * _flops2(c, c["n"], c["nedge"], c["data"]),
                "bytes": c["nprop"] * 80 + c["data"] * min(c["nbins"] ** 2, c["side"] ** 2) * 16}
    if kind == "fields":
        f = _flops2(c, c["n"], c["nedge"], 1) + _flops2(c, c["n2"], c["nedge"] // 2, 1)
        return {"flops": c["nprop"] * f,
                "bytes": c["nprop"] * 80 + 2 * min(c["nbins"] ** 2, c["side"] ** 2) * 16}
    if kind == "chain":
        k = _chain1(c)
        f = _flops1(k, _inputs1(dict(k, nprop=1, side=64), 0), c["walkers"], 1)
        return {"flops": c["steps"] * f,
                "bytes": c["steps"] * c["walkers"] * (4 * c["knots"] + 12)}
    h, i = c["hidden"], c["inputs"]
    macs = i * h + 2 * h * h + h
    return {"flops": 2.0 * macs * (3 * c["iters"] * c["batch"] + c["rows"]),
            "bytes": c["iters"] * (c["batch"] * (4.0 * i + 8) + 28.0 * macs)}


def _flops1(c, q, nprop, ndata):
    n, ni = c["n"], c["ninterp"]
    total = 0.0
    for bm in q["beams"]:
        for neg in (False, True):
            w, ie = _terms1(bm, c["hist"], neg)
            if ie.size:
                x = np.abs(_nodes1(q["kp"], 1.0 / ie.min(), neg, ni))
                a = x[:, None] * ie[None, :]
                total += 25.0 * np.count_nonzero((a >= q["kp"][0]) & (a < q["kp"][-1]))
        fft = 2.5 * n * math.log2(n)
        total += 15.0 * n + fft + ndata * (20.0 * n + fft + 6.0 * n)
    return nprop * total


def _flops2(c, n, nedge, ndata):
    q = _inputs2(dict(c, nprop=1, side=64, data=1), 0)
    B = _beam2(q["b1"], q["b2"], c.get("hist", 100))
    m = _Model2(q, q["theta0"])
    rr = _range2(m, B, q["sig"], None)
    a1 = _axis2(n, rr[0], rr[1])[0]
    rows = np.abs(a1[a1 != 0])
    terms = 0
    for s in B.values():
        a = rows[:, None] * s["ie1"][None, :]
        terms += np.count_nonzero((a >= q["kp"][0]) & (a < q["kp"][-1]) & (rows[:, None] < q["kp"][-1] * s["max1"]))
    # a term meets the columns of its own band-2 sign
    cells = terms * (n + nedge) * (1.0 if len(B) == 1 else 0.5)
    fft = 5.0 * n * n * math.log2(n)
    return 25.0 * cells + fft + ndata * (20.0 * n * n + fft + 2.0 * n * n)


# --------------------------------------------------- float64 restatements
def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "like1":
        ll = _exact1(c, _inputs1(c, seed))
        return (np.float64(ll[0]), None) if c["nprop"] == 1 else (ll, None)
    if kind == "pd1":
        q = _inputs_pd1(c, seed)
        th = np.concatenate([q["kv"], [1.0]])[None, :]
        G = _grid1(c["n"], q["lo"], q["hi"])
        R = _rgrid1(G, q["kp"], q["bm"], c["hist"], c["ninterp"], th)
        p, info = _pd1(G, R, q["noise"], 0)
        return {"pd": p, "minflux": np.float64(info["minflux"]), "dflux": np.float64(G["dflux"])}
    if kind == "like2":
        return _exact2(c, _inputs2(c, seed), c["n"], c["nedge"], 0), None
    if kind == "fields":
        q = _inputs2(c, seed, 2)
        return (_exact2(c, q, c["n"], c["nedge"], 0) +
                _exact2(c, q, c["n2"], c["nedge"] // 2, 1), None)
    return None  # a chain and a bf16 training run have no float64 value


def _natural(x, y):
    """Natural cubic spline through y [..., n] at x [n]: per interval
    (y, b, c, d), the tridiagonal system by forward and back substitution."""
    x = np.asarray(x, np.float64)
    h = np.diff(x)
    n = x.size
    s = np.diff(y, axis=-1) / h
    g = 3.0 * np.diff(s, axis=-1)
    diag = 2.0 * (h[1:] + h[:-1])
    N = n - 2
    z = np.moveaxis(g, -1, 0).copy()
    al = np.empty(N)
    ga = np.empty(N)
    al[0] = diag[0]
    for i in range(N):
        if i:
            al[i] = diag[i] - h[i] * ga[i - 1]
            z[i] -= ga[i - 1] * z[i - 1]
        ga[i] = h[i + 1] / al[i]
    cc = np.zeros((n,) + z.shape[1:])
    for i in range(N - 1, -1, -1):
        cc[i + 1] = z[i] / al[i] - (ga[i] * cc[i + 2] if i < N - 1 else 0.0)
    cc = np.moveaxis(cc, 0, -1)
    b = s - h * (cc[..., 1:] + 2.0 * cc[..., :-1]) / 3.0
    d = np.diff(cc, axis=-1) / (3.0 * h)
    return np.stack([y[..., :-1], b, cc[..., :-1], d], -1)


def _cubic(x, coef, v):
    """Spline (one row) at v, the end intervals extended."""
    k = np.clip(np.searchsorted(x, v, side="right") - 1, 0, x.size - 2)
    dl = v - x[k]
    q = coef[k]
    return q[..., 0] + dl * (q[..., 1] + dl * (q[..., 2] + dl * q[..., 3]))


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


# ---- 1D
def _terms1(pix, hist, neg):
    v = np.sort(-pix[pix < -1e-5] if neg else pix[pix > 1e-5])
    if v.size == 0:
        return np.empty(0), np.empty(0)
    if not hist or np.count_nonzero(pix > 1e-5) < 20:
        return np.ones(v.size), 1.0 / v
    lo, hi = math.log2(v[0]) - HISTPAD, math.log2(v[-1]) + HISTPAD
    b = ((np.log2(v) - lo) / ((hi - lo) / hist)).astype(int)
    cnt = np.bincount(b, minlength=hist)
    tot = np.bincount(b, weights=v, minlength=hist)
    k = cnt > 0
    return cnt[k].astype(float), 1.0 / (tot[k] / cnt[k])


def _nodes1(kp, maxbeam, neg, ni):
    i = np.arange(ni)
    if not neg:
        lo, hi = kp[0] * 1e-5, kp[-1] * maxbeam
        hi -= 0.001 * (hi - lo) / (ni - 1)
        return lo * np.exp2(i * (math.log2(hi / lo) / (ni - 1)))
    hi, lo = -kp[0] * 1e-5, -kp[-1] * maxbeam
    d = 0.001 * (hi - lo) / (ni - 1)
    lo, hi = lo + d, hi - d
    return hi * np.exp2((ni - 1 - i) * (math.log2(lo / hi) / (ni - 1)))


def _grid1(n, lo, hi):
    """The wrapped flux grid of R."""
    lo = min(lo, 0.0)
    if lo == 0.0:
        return {"n": n, "wrap": n - 1, "dflux": hi / (n - 1), "low": 0.0}
    d = (hi - lo) / (n - 1)
    d = hi / (n - math.floor(-lo / d) - 1.0)
    w = int(hi / d + 0.9999999999)
    return {"n": n, "wrap": w, "dflux": d, "low": (w + 1) * d - n * d}


def _rgrid1(G, kp, pix, hist, ni, theta):
    """R dflux on the wrapped grid for rows of log10 knot values: [P, n]."""
    K, P = kp.size, theta.shape[0]
    lk = np.log2(kp)
    spl = _natural(lk, math.log2(10.0) * theta[:, :K].astype(np.float64))
    n, wrap, d = G["n"], G["wrap"], G["dflux"]
    R = torch.zeros(P, n, dtype=torch.float64, device=DEV)
    for neg in (False, True):
        w, ie = _terms1(pix, hist, neg)
        if ie.size == 0 or (neg and G["low"] >= 0.0):
            continue
        vmax = np.abs(pix[pix < -1e-5]).max() if neg else pix.max()
        x = _nodes1(kp, vmax, neg, ni)
        S = _t(spl)
        acc = torch.zeros(P, ni, dtype=torch.float64, device=DEV)
        arg = np.abs(x)[:, None] * ie[None, :]
        u = np.log2(np.abs(x))[:, None] + np.log2(ie)[None, :]
        ok = (arg >= kp[0]) & (arg < kp[-1])
        kk = np.clip(np.searchsorted(lk, u, side="right") - 1, 0, K - 2)
        tk, tu, tok = _t(kk), _t(u - lk[kk]), _t(ok.astype(np.float64))
        for j in range(ie.size):
            if not ok[:, j].any():
                continue
            q = S[:, tk[:, j]]
            dl = tu[:, j]
            e = q[..., 0] + dl * (q[..., 1] + dl * (q[..., 2] + dl * q[..., 3]))
            acc += tok[:, j] * (w[j] * ie[j]) * torch.exp2(e)
        acc = (acc * (PIX / 3600.0) ** 2).cpu().numpy()
        y = np.where(acc > 0, np.log2(np.where(acc > 0, acc, 1.0)), SMALLLOG)
        co = _natural(x, y)
        if not neg:
            lo, hi = int(x[0] / d + 0.9999999999999999), min(int(x[-1] / d), wrap)
            off = 0.0
        else:
            lo = max(int((x[0] - G["low"]) / d + wrap + 1 + 0.9999999999999999), wrap + 1)
            hi = min(int((x[-1] - G["low"]) / d + wrap + 1), n - 1)
            off = G["low"] - (wrap + 1) * d
        i = np.arange(lo, hi + 1)
        f = i * d + off
        k = np.clip(np.searchsorted(x, f, side="right") - 1, 0, ni - 2)
        q = _t(co)[:, _t(k)]
        dl = _t(f - x[k])
        e = q[..., 0] + dl * (q[..., 1] + dl * (q[..., 2] + dl * q[..., 3]))
        R[:, lo:hi + 1] = torch.exp2(e) * d
    return R


def _wrapped1(G, R, sigma):
    """The wrapped P(D) of every row for one noise level, and var(R)."""
    n, wrap, d, low = G["n"], G["wrap"], G["dflux"], G["low"]
    i = np.arange(n)
    cf = np.where(i <= wrap, i * d, (i - wrap - 1) * d + low)
    w = np.ones(n)
    w[0], w[wrap] = 0.0, 0.5
    mn = (R * _t(w * cf)).sum(1)
    var = (R * _t(w * cf * cf)).sum(1)
    if wrap < n - 1:
        p = 0.5 * low * R[:, wrap - 1]
        mn, var = mn - p, var - low * p
    shift = torch.where((torch.sqrt(var) > d) & (mn.abs() > d), -mn, torch.zeros_like(mn))
    rt = torch.fft.rfft(R)
    k = torch.arange(rt.shape[1], device=DEV, dtype=torch.float64)
    fl = 2 * math.pi / (n * d)
    amp = torch.exp(rt.real - rt.real[:, :1]) * torch.exp(-0.5 * (sigma * fl * k) ** 2)
    ph = rt.imag - (shift * fl)[:, None] * k
    P = torch.polar(amp, ph)
    P[:, 0] = 1.0
    if n % 2 == 0:
        P[:, -1] = P[:, -1].real.to(P.dtype)
    return torch.clamp(torch.fft.irfft(P, n) * n, min=0.0), var


def _split(p, bot, top, f1, f2, f3, low_rule):
    """The split search: the minimum in [bot, top], kept when it is reached
    monotonically over 17 values, else the first value below the jitter
    level from the top."""
    if bot < 0 or bot > top or top >= p.size:
        return None
    mi = bot + int(np.argmin(p[bot:top + 1]))
    mv, peak = p[mi], p.max()
    if mv > f2 * peak:
        return None
    if mi > 17:
        pre = p[mi - 17:mi]
        if np.all(np.diff(pre) < 0):
            return mi
        jit = 1.1 * (pre.sum() + mv) / 18
    else:
        jit = f1 * peak
        if mv > jit:
            return mi
    if mv <= 0:
        lo = bot if mi < bot else low_rule(mi)
        hi = top - 3 if mi > top - 3 else mi + 3
        mv = max([mv] + [p[j] for j in range(max(lo, 0), hi)])
    if mv > 0:
        jit = min(f3 * mv, jit)
    if bot >= top or p[top] < jit:
        return None
    hit = np.nonzero(p[bot:top] < jit)[0]
    return bot + int(hit[-1]) + 1 if hit.size else None


def _finish1(G, p, var, sigma):
    """Split, normalisation and mean of one wrapped P(D) row."""
    n, wrap, d, low = G["n"], G["wrap"], G["dflux"], G["low"]
    sp = math.sqrt(var + sigma * sigma)
    sn = sigma if 9 * sigma * sigma > var else sp
    bot = int(2.5 * sp / d)
    top = wrap if 2.5 * sp > abs(low) else int(-(2.5 * sn + low) / d + wrap + 1)
    s = _split(p, bot, top, 5e-14, 1e-5, 5.0, lambda m: m - 3)
    if s is None:
        return None, math.nan
    q = np.concatenate([p[s:], p[:s]])
    q = q / ((q.sum() - 0.5 * (q[0] + q[-1])) * d)
    w = np.arange(n, dtype=np.float64)
    w[-1] *= 0.5
    return q, -(w * q).sum() * d * d


def _pd1(G, R, sigma, row):
    p, var = _wrapped1(G, R, sigma)
    q, mf = _finish1(G, p[row].cpu().numpy(), float(var[row]), sigma)
    return q, {"minflux": mf}


def _bins1(m, nbins):
    d = m.ravel() - m.mean()
    lo = d.min()
    step = (d.max() - lo) / (nbins - 1)
    cnt = np.bincount(((d - lo) * (1.0 / step) + 0.5).astype(np.int64), minlength=nbins)
    return lo, step, cnt


def _log2p(q):
    return np.where(q > 0, np.log2(np.where(q > 0, q, 1.0)), SMALLLOG)


def _exact1(c, q):
    th = q["theta"]
    out = np.zeros(th.shape[0])
    for b, pix in enumerate(q["beams"]):
        pos = pix[pix > 1e-5]
        neg = -pix[pix < -1e-5]
        data, lo, hi = [], math.inf, -math.inf
        for m in q["maps"][b]:
            if c["binned"]:
                x0, dx, cnt = _bins1(m, c["nbins"])
                data.append((x0 + np.arange(cnt.size) * dx, cnt))
                lo, hi = min(lo, x0), max(hi, x0 + (c["nbins"] - 1) * dx)
            else:
                v = m.ravel() - m.mean()
                data.append((v, None))
                lo, hi = min(lo, v.min()), max(hi, v.max())
        smax = max(q["sig"][b])
        rlo = -1.05 * q["kp"][-1] * neg.max() if neg.size else 0.0
        rhi = 1.05 * q["kp"][-1] * pos.max() + NZEROPAD * smax
        if neg.size:
            rlo = min(rlo, lo)
        rhi = max(rhi, hi)
        G = _grid1(c["n"], rlo, rhi)
        n, d = c["n"], G["dflux"]
        R = _rgrid1(G, q["kp"], pix, c["hist"], c["ninterp"], th)
        for (f, cnt), s in zip(data, q["sig"][b]):
            npix = f.size if cnt is None else cnt.sum()
            off = -0.5 * npix * (math.log(2 * math.pi * s * s) + 1.0)
            p, var = _wrapped1(G, R, s)
            p, var = p.cpu().numpy(), var.cpu().numpy()
            for r in range(th.shape[0]):
                pr, mf = _finish1(G, p[r], float(var[r]), s)
                if pr is None:
                    out[r] = math.nan
                    continue
                lp = _log2p(pr)
                t = np.clip((f - mf) / d, 0.0, n - 1.0)
                k = np.minimum(t.astype(np.int64), n - 2)
                t = t - k
                v = (1.0 - t) * lp[k] + t * lp[k + 1]
                v = np.where(f < mf, lp[0], np.where(f > mf + (n - 2) * d, lp[-1], v))
                out[r] += math.log(2.0) * (v if cnt is None else v * cnt).sum() - off
    return out


# ---- two bands
class _Model2:
    """Knot counts and the log-normal colour curves of one parameter row."""

    def __init__(self, q, theta):
        K, ns, no = q["kp"].size, q["sk"].size, q["ok"].size
        t = np.asarray(theta, np.float64)
        self.kp, self.lk = q["kp"], np.log2(q["kp"])
        self.spl = _natural(self.lk, math.log2(10.0) * t[:K])
        self.sig = self._curve(q["sk"], t[K:K + ns])
        self.off = self._curve(q["ok"], t[K + ns:K + ns + no])

    @staticmethod
    def _curve(x, y):
        if x.size == 1:
            return lambda f: np.full(np.shape(f), y[0])
        if x.size == 2:
            return lambda f: y[0] + (np.clip(f, x[0], x[1]) - x[0]) / (x[1] - x[0]) * (y[1] - y[0])
        co = _natural(x, y)
        return lambda f: np.where(f <= x[0], y[0], np.where(
            f >= x[-1], y[-1], _cubic(x, co, np.clip(f, x[0], x[-1]))))

    def counts(self, f):
        return np.exp2(_cubic(self.lk, self.spl, np.log2(f)))

    def maxflux2(self):
        """Band-2 flux three sigma above the mode of the colour at the last
        knot (Brent's method, stopped at a relative bracket of 1e-3)."""
        kv = self.kp[-1]
        mu, sig = float(self.off(kv)), float(self.sig(kv))
        mode = mu - sig * sig
        target = math.exp(0.5 * sig * sig - mu) / sig * math.exp(-4.5)

        def F(u):
            return math.exp(-0.5 * ((u - mu) / sig) ** 2) / sig * math.exp(-u) - target
        step = math.log(math.exp(mode) + 2 * sig) - mode
        while F(mode + step) >= 0.0:
            step *= 1.5
        return kv * math.exp(_brent(F, mode, mode + step))


def _brent(F, a, b):
    """Brent (1973, ch. 4), until the bracket is below 1e-3 of the root."""
    eps = np.finfo(float).eps
    c, fa, fb = b, F(a), F(b)
    fc = fb
    d = e = b - a
    for _ in range(20):
        fresh = False
        if (fb < 0) == (fc < 0):
            fresh, c, fc = True, a, fa
            d = e = b - a
        if abs(fc) < abs(fb):
            fresh = True
            a, b, c = b, c, b
            fa, fb, fc = fb, fc, fb
        tol, m = 0.5 * eps * abs(b), 0.5 * (c - b)
        if fb == 0 or abs(m) <= tol:
            return b
        if abs(e) < tol or abs(fa) <= abs(fb):
            d = e = m
        else:
            s = fb / fa
            if fresh:
                p, q = 2 * m * s, 1 - s
            else:
                u, r = fa / fc, fb / fc
                p = s * (2 * m * u * (u - r) - (b - a) * (r - 1))
                q = (u - 1) * (r - 1) * (s - 1)
            if p > 0:
                q = -q
            else:
                p = -p
            if 2 * p < min(3 * m * q - abs(tol * q), abs(e * q)):
                e, d = d, p / q
            else:
                d = e = m
        a, fa = b, fb
        b += d if abs(d) > tol else math.copysign(tol, m)
        fb = F(b)
        o = a if (fb < 0) == (fc < 0) else c
        lo = min(abs(b), abs(o)) if (b > 0) == (o > 0) else 0.0
        if abs(b - o) < 1e-3 * lo:
            return b
    return b


def _beam2(p1, p2, hist):
    """Sign components (pp, pn, np, nn = 0 .. 3) as weight / inverse band-1
    beam / log beam ratio lists."""
    out = {}
    a1, a2 = np.abs(p1).ravel(), np.abs(p2).ravel()
    use = (a1 > 1e-6) & (a2 > 1e-6)
    sgn = np.where(p1.ravel() > 0, 0, 2) + np.where(p2.ravel() > 0, 0, 1)
    for s in range(4):
        k = use & (sgn == s)
        if not k.any():
            continue
        v1, v2 = a1[k], a2[k]
        r = {"max1": v1.max(), "max2": v2.max()}
        if v1.size >= 30:
            b = []
            for v in (v1, v2):
                lo, hi = math.log2(v.min()) - HISTPAD, math.log2(v.max()) + HISTPAD
                b.append(((np.log2(v) - lo) * (hist / (hi - lo))).astype(int))
            t = b[0] * hist + b[1]
            cnt = np.bincount(t, minlength=hist * hist)
            m = cnt > 0
            r["w"] = cnt[m].astype(float)
            r["ie1"] = r["w"] / np.bincount(t, weights=v1, minlength=hist * hist)[m]
            ie2 = r["w"] / np.bincount(t, weights=v2, minlength=hist * hist)[m]
            r["lr"] = np.log(ie2 / r["ie1"])
        else:
            r["w"], r["ie1"], r["lr"] = np.ones(v1.size), 1.0 / v1, np.log(v1 / v2)
        out[s] = r
    return out


def _range2(m, B, sig, data):
    k1, k2 = m.kp[-1], m.maxflux2()
    lo1 = -k1 * max([B[s]["max1"] for s in (2, 3) if s in B], default=0.0)
    hi1 = k1 * max([B[s]["max1"] for s in (0, 1) if s in B], default=0.0)
    lo2 = -k2 * max([B[s]["max2"] for s in (1, 3) if s in B], default=0.0)
    hi2 = k2 * max([B[s]["max2"] for s in (0, 2) if s in B], default=0.0)
    r = [1.1 * lo1, 1.1 * hi1 + NZEROPAD * sig[0], 1.1 * lo2, 1.1 * hi2 + NZEROPAD * sig[1]]
    if data is not None:
        if 2 in B or 3 in B:
            r[0] = min(r[0], data[0])
        r[1] = max(r[1], data[1])
        if 1 in B or 3 in B:
            r[2] = min(r[2], data[2])
        r[3] = max(r[3], data[3])
    return r


def _axis2(n, lo, hi):
    d = (hi - lo) / (n - 1)
    i = np.arange(n, dtype=np.float64)
    if lo >= 0.0:
        return i * d + lo, d
    d = hi / (n - math.floor(-lo / d) - 1.0)
    w = int(hi / d + 0.999999999)
    return np.where(i <= w, i * d, i * d - n * d), d


def _rows2(m, B, rowf, colf):
    """R (without the flux steps) at rowf x colf, one cell per pair."""
    neg = 2 in B or 3 in B
    R = torch.zeros(rowf.size, colf.size, dtype=torch.float64, device=DEV)
    nz = colf != 0
    lf2 = _t(np.where(nz, np.log(np.abs(np.where(nz, colf, 1.0))), 0.0))
    inv = _t(np.where(nz, 1.0 / np.abs(np.where(nz, colf, 1.0)), 0.0))
    pref = (PIX / 3600.0) ** 2 / math.sqrt(2 * math.pi)
    for s, t in B.items():
        rows = (rowf > 0) if s < 2 else ((rowf < 0) & neg)
        cols = _t(((colf > 0) if s % 2 == 0 else (colf < 0)).astype(np.float64))
        f1 = np.abs(rowf)
        for j in range(t["w"].size):
            a = f1 * t["ie1"][j]
            ok = rows & (f1 < m.kp[-1] * t["max1"]) & (a >= m.kp[0]) & (a < m.kp[-1])
            if not ok.any():
                continue
            r = np.nonzero(ok)[0]
            a = a[r]
            isg = 1.0 / m.sig(a)
            c0 = t["w"][j] * t["ie1"][j] * isg * m.counts(a) * pref
            c1 = np.log(f1[r]) + m.off(a) - t["lr"][j]
            z = (lf2[None, :] - _t(c1)[:, None]) * _t(isg)[:, None]
            R[_t(r)] += _t(c0)[:, None] * torch.exp(-0.5 * z * z) * cols
    return R * inv


def _exact2(c, q, n, nedge, field):
    B = _beam2(q["b1"], q["b2"], c.get("hist", 100))
    nb = c["nbins"]
    data, rng = [], [math.inf, -math.inf] * 2
    for m1, m2 in q["maps"][field]:
        e = []
        for band, m in enumerate((m1, m2)):
            d = m.ravel() - m.mean()
            lo = d.min()
            st = (d.max() - lo) / (nb - 1)
            e.append((lo, st, ((d - lo) * (1.0 / st) + 0.5).astype(np.int64)))
            rng[2 * band] = min(rng[2 * band], lo)
            rng[2 * band + 1] = max(rng[2 * band + 1], lo + (nb - 1) * st)
        t, cnt = np.unique(e[0][2] * nb + e[1][2], return_counts=True)
        f1 = e[0][0] + (t // nb) * e[0][1]
        f2 = e[1][0] + (t % nb) * e[1][1]
        data.append((_t(f1), _t(f2), _t(cnt.astype(float)), m1.size))
    rr = _range2(_Model2(q, q["theta0"]), B, q["sig"], rng)
    a1, d1 = _axis2(n, rr[0], rr[1])
    a2, d2 = _axis2(n, rr[2], rr[3])
    # edge fluxes below the first grid step: logarithmic in band 1, linear
    # in band 2
    i = np.arange(nedge)
    lg = -math.log(1e-9) / (nedge - 1)
    E1 = d1 * 1e-9 * np.exp(i * lg)
    st2 = (d2 - d2 * 1e-9) / (nedge - 1)
    E2 = d2 * 1e-9 + i * st2
    trap = np.ones(nedge)
    trap[0] = trap[-1] = 0.5
    w1 = _t(trap * E1 * lg / (d1 - d1 * 1e-9))
    w2 = _t(trap * st2 / (d2 - d2 * 1e-9))
    wt = np.ones(n)
    wt[0] = wt[-1] = 0.5
    s1, s2 = q["sig"]
    out = np.zeros(q["theta"].shape[0])
    rows, cols = np.concatenate([a1, E1]), np.concatenate([a2, E2])
    off = [-float(dd[3]) * (math.log(2 * math.pi * s1 * s2) + 1.0) for dd in data]
    for r in range(out.size):
        F = _rows2(_Model2(q, q["theta"][r]), B, rows, cols) * (d1 * d2)
        R = F[:n, :n].clone()
        R[0, 1:] = w1 @ F[n:, 1:n]
        R[1:, 0] = F[1:n, n:] @ w2
        R[0, 0] = w1 @ F[n:, n:] @ w2
        del F
        out[r] = _like2_row(R, a1, a2, d1, d2, wt, s1, s2, data, off)
    return out


def _like2_row(R, a1, a2, d1, d2, wt, s1, s2, data, off):
    n = a1.size
    W1, W2 = _t(wt), _t(wt)
    rs, cs = R @ W2, W1 @ R
    m1, v1 = float((W1 * _t(a1) * rs).sum()), float((W1 * _t(a1 * a1) * rs).sum())
    m2, v2 = float((W2 * _t(a2) * cs).sum()), float((W2 * _t(a2 * a2) * cs).sum())
    sh1 = -m1 if math.sqrt(v1) > d1 and abs(m1) > d1 else 0.0
    sh2 = -m2 if math.sqrt(v2) > d2 and abs(m2) > d2 else 0.0
    rt = torch.fft.fft(torch.fft.rfft(R, dim=1), dim=0)
    k1 = np.arange(n)
    k1 = np.where(k1 < n // 2 + 1, k1, k1 - n).astype(float)
    k2 = np.arange(n // 2 + 1, dtype=float)
    u1, u2 = _t(2 * math.pi / (n * d1) * k1)[:, None], _t(2 * math.pi / (n * d2) * k2)[None, :]
    amp = torch.exp((rt.real - rt.real[0, 0]) - 0.5 * ((s1 * u1) ** 2 + (s2 * u2) ** 2))
    P = torch.polar(amp, rt.imag - sh1 * u1 - sh2 * u2)
    P[0, 0] = 1.0
    p = torch.fft.irfft(torch.fft.ifft(P, dim=0) * n, n, dim=1) * n
    p = torch.clamp(p, min=0.0)
    del P, rt, amp

    def split(marg, var, s, d):
        sp = math.sqrt(var + s * s)
        sn = s if 9 * s * s > var else sp
        return _split(marg, int(2.25 * sp / d), n - int(2.25 * sn / d) - 1, 5e-14, 1.5e-5,
                      5.0, lambda m: m - 3 if m >= 3 else m)
    x1 = split((p @ W2).cpu().numpy(), v1, s1, d1)
    x2 = split((W1 @ p).cpu().numpy(), v2, s2, d2)
    if x1 is None or x2 is None:
        return math.nan
    p = torch.roll(p, (-x1, -x2), (0, 1))
    tot = float(W1 @ p @ W2) * d1 * d2
    p = p / tot
    j = _t(np.arange(n, dtype=float))
    f1 = -float((W1 * j * (p @ W2)).sum()) * d1 * d1 * d2
    f2 = -float((W2 * j * (W1 @ p)).sum()) * d1 * d2 * d2
    lp = torch.where(p > 0, torch.log2(torch.where(p > 0, p, torch.ones_like(p))),
                     torch.full_like(p, SMALLLOG))
    ll = 0.0
    for (b1, b2, cnt, _), o in zip(data, off):
        def place(f, f0, d):
            """Cell and weight of the upper neighbour, the edges clamped."""
            t = (f - f0) / d
            k = t.to(torch.int64)
            t = t - k
            t = torch.where(k > n - 2, torch.ones_like(t), t)
            k = torch.clamp(k, max=n - 2)
            lo, hi = f < f0, f > f0 + (n - 1) * d
            k = torch.where(lo, torch.zeros_like(k), torch.where(hi, torch.full_like(k, n - 2), k))
            t = torch.where(lo, torch.zeros_like(t), torch.where(hi, torch.ones_like(t), t))
            return k, t, lo | hi
        i1, t1, o1 = place(b1, f1, d1)
        i2, t2, o2 = place(b2, f2, d2)
        # beyond one band's range the other band's lower cell is read as is
        t2 = torch.where(o1 & ~o2, torch.zeros_like(t2), t2)
        t1 = torch.where(o2 & ~o1, torch.zeros_like(t1), t1)
        v = (1 - t1) * ((1 - t2) * lp[i1, i2] + t2 * lp[i1, i2 + 1]) + \
            t1 * ((1 - t2) * lp[i1 + 1, i2] + t2 * lp[i1 + 1, i2 + 1])
        ll += math.log(2.0) * float((cnt * v).sum()) - o
    return ll
