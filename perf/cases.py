"""The work that users of this engine have it do, at sizes over its real range.

Each case is one call pattern through the public Python face of the engine:

  chain      Engine.price: one parameter set, an option chain (or one option)
  book       Engine.price_batch: many sets with uneven chains, host to host
  graph      Engine.prepare_batch once, then Batch.launch and Batch.collect
  serve      Engine.server: a burst of requests submitted, then waited for
  calibrate  Engine.calibration: the objective and Jacobian at a point and
             the objective at a trial point, a Levenberg-Marquardt step
  swift      Engine.swift_batch: European surfaces with their gradients

``listed`` has the named cases, ``draw`` one more of the same ranges,
``prepare`` a case's inputs from a seed, ``run`` one pass, ``work`` what a
pass cannot do without, and ``exact`` the same results in 64 bits, written
here in plain torch and numpy: the generator, the inverse normal, the QE
scheme and the contracts step by step, the geometric average's affine
recursion, and the SWIFT sums as matrix products.
"""
import math

import numpy as np
import torch

from hestonexotics_gb300 import ASIAN, EUROPEAN, FP32, FP64, STEP_GRID, STEP_REFERENCE, Config, Engine, Options, Params, Request

S0 = 100.0
STEPS_PER_YEAR = 252.0
CHAIN = (1 / 12, 1 / 4, 1 / 2, 3 / 4, 1.0, 1.5, 2.0, 3.0)   # the single chain's maturities, years


# ------------------------------------------------------------------- cases

def listed():
    return [
        # one quick quote, the smallest call: latency of the steps, the launches and the host path
        dict(name="quote-fp64", kind="chain", precision="fp64", model="plain", paths=5000, steps=60, maturities=1,
             longest=1.0, strikes=1, payoffs="asian", cv=False),
        # the plain Asian request at its usual size, in both forms
        dict(name="asian-fp64", kind="chain", precision="fp64", model="plain", paths=65536, steps=252, maturities=1,
             longest=1.0, strikes=1, payoffs="asian", cv=False),
        dict(name="asian-fp32", kind="chain", precision="fp32", model="plain", paths=65536, steps=252, maturities=1,
             longest=1.0, strikes=1, payoffs="asian", cv=False),
        # a whole option chain on the daily grid, odd path count, the default (FP64) form
        dict(name="chain-fp64", kind="chain", precision="fp64", model="drawn", paths=100003, steps=0, maturities=8,
             longest=3.0, strikes=50, payoffs="both", cv=False),
        # the same chain at the full path count in the batched FP32 form
        dict(name="chain-fp32", kind="chain", precision="fp32", model="drawn", paths=1 << 20, steps=0, maturities=8,
             longest=3.0, strikes=50, payoffs="both", cv=False),
        # high vol-of-vol: most steps take the exponential branch
        dict(name="feller-fp64", kind="chain", precision="fp64", model="feller", paths=65537, steps=0, maturities=8,
             longest=3.0, strikes=50, payoffs="both", cv=False),
        # fewer paths to the same error: Asian chain with the geometric control variate
        dict(name="chain-cv-fp32", kind="chain", precision="fp32", model="drawn", paths=200000, steps=0, maturities=8,
             longest=3.0, strikes=50, payoffs="asian", cv=True),
        # end-of-day book: 64 sets with uneven chains, path counts spread over a factor of 256
        dict(name="book-fp32", kind="book", precision="fp32", sets=64, options=400, paths_lo=10, paths_hi=18, book=2),
        # a book re-priced with one graph launch, the FP64 form
        dict(name="graph-fp64", kind="graph", precision="fp64", sets=12, options=150, paths_lo=9, paths_hi=14, book=5),
        # a burst at the server: single-set requests of 1 to 400 options at the path count of a target error
        dict(name="serve-fp32", kind="serve", precision="fp32", sets=32, options=400, paths=40000, book=3),
        # one Levenberg-Marquardt step of the calibration: 8 expiries of 5 quotes
        dict(name="calibrate", kind="calibrate", expiries=8, strikes=5, trunc=1e-7),
        # European surfaces with gradients for a set of candidate parameters
        dict(name="swift-surface", kind="swift", sets=256, expiries=8, strikes=50, trunc=1e-7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "chain", "chain", "book", "graph", "serve", "calibrate", "swift"])
    precision = rng.choice(["fp64", "fp32"])
    budget = 1.2e9 if precision == "fp64" else 1.2e10   # path-steps
    if kind == "chain":
        case = dict(kind=kind, precision=precision, model=rng.choice(["plain", "drawn", "feller"]),
                    steps=rng.choice([0, 0, _log_int(rng, 24, 400)]), maturities=rng.choice([1, 2, 3, 5, 8]),
                    longest=round(rng.uniform(0.25, 4.0), 3), strikes=_log_int(rng, 1, 100),
                    payoffs=rng.choice(["asian", "european", "both"]), cv=rng.random() < 0.2, paths=1)
        steps = max(1.0, work(case)["flops"] / _FLOPS)
        case["paths"] = _log_int(rng, 1000, min(1 << 20, max(2000, budget / steps)))
        return case
    if kind in ("book", "graph"):
        sets = _log_int(rng, 2, 48)
        hi = rng.randint(12, 18) if precision == "fp32" else rng.randint(10, 14)
        return dict(kind=kind, precision=precision, sets=sets, options=_log_int(rng, 10, 400), paths_lo=max(7, hi - 8),
                    paths_hi=hi, book=rng.randrange(1 << 20))
    if kind == "serve":
        return dict(kind=kind, precision="fp32", sets=_log_int(rng, 2, 48), options=_log_int(rng, 2, 400),
                    paths=_log_int(rng, 16384, 80000), book=rng.randrange(1 << 20))
    if kind == "calibrate":
        return dict(kind=kind, expiries=rng.randint(1, 12), strikes=rng.randint(1, 20), trunc=rng.choice([1e-7, 1e-10]))
    return dict(kind=kind, sets=_log_int(rng, 1, 300), expiries=rng.randint(1, 8), strikes=_log_int(rng, 5, 80),
                trunc=rng.choice([1e-7, 1e-10]))


# ------------------------------------------------------------------ inputs

def _params(model, g):
    """(v0, theta, rho, kappa, sigma, r, q)."""
    if model == "drawn":
        return (g.uniform(0.01, 0.09), g.uniform(0.01, 0.09), g.uniform(-0.9, -0.1), g.uniform(0.5, 5.0),
                g.uniform(0.1, 1.0), g.uniform(0.0, 0.05), 0.0)
    near = g.uniform(0.95, 1.05, 4)
    if model == "feller":
        return (0.04 * near[0], 0.04 * near[1], -0.9, 0.5 * near[2], 1.0 * near[3], 0.02, 0.0)
    return (0.04 * near[0], 0.04 * near[1], -0.7, 1.5 * near[2], 0.5 * near[3], 0.02, 0.0)


def _daily(T):
    return np.maximum(5, np.rint(np.asarray(T) * STEPS_PER_YEAR)) / STEPS_PER_YEAR


def _maturities(case):
    n, longest = case["maturities"], case["longest"]
    T = np.array(CHAIN) if n == len(CHAIN) and longest == CHAIN[-1] else longest * np.arange(1, n + 1) / n
    return T if case["steps"] else _daily(T)


def _book(case):
    """The shape of a book: per set its maturities and path counts per option; the same for every seed."""
    g = np.random.default_rng(case["book"])
    out = []
    for _ in range(case["sets"]):
        n = int(g.integers(1 if case["kind"] == "serve" else min(10, case["options"]), case["options"] + 1))
        T = _daily(g.uniform(0.02, 5.0, n))
        if case["kind"] == "serve":
            paths = np.full(n, case["paths"], dtype=np.uint64)
        else:
            u = np.unique(T)
            paths = np.rint(2.0 ** g.uniform(case["paths_lo"], case["paths_hi"], len(u))).astype(np.uint64)[
                np.searchsorted(u, T)]
        out.append((T, paths))
    return out


def _requests(case, seed):
    """Plain requests (params, strikes, T, payoff, paths, seed, stream) of a Monte Carlo case, and its step count
    per maturity (0: the daily grid)."""
    g = np.random.default_rng([seed, 17])
    if case["kind"] == "chain":
        T, K, P = [], [], []
        strikes = np.geomspace(0.6 * S0, 1.6 * S0, case["strikes"]) if case["strikes"] > 1 else np.array([S0])
        strikes = strikes * g.uniform(0.99, 1.01, len(strikes))
        kinds = {"asian": (ASIAN,), "european": (EUROPEAN,), "both": (ASIAN, EUROPEAN)}[case["payoffs"]]
        for t in _maturities(case):
            for k in kinds:
                T.append(np.full(len(strikes), t))
                K.append(strikes)
                P.append(np.full(len(strikes), k))
        T, K, P = np.concatenate(T), np.concatenate(K), np.concatenate(P)
        n = np.full(len(T), case["paths"], dtype=np.uint64)
        return [(_params(case["model"], g), K, T, P, n, int(g.integers(1 << 32)), 0)], case["steps"]
    reqs = []
    for s, (T, n) in enumerate(_book(case)):
        K = S0 * np.exp(g.uniform(math.log(0.6), math.log(1.6), len(T)))
        P = np.where(g.random(len(T)) < 0.75, ASIAN, EUROPEAN)
        reqs.append((_params("drawn", g), K, T, P, n, int(g.integers(1 << 32)), s))
    return reqs, 0


def _surfaces(case, seed):
    """(parameters, spot, [(expiry, strikes)]) of a calibration's points or of a batch of surfaces."""
    g = np.random.default_rng([seed, 29])
    if case["kind"] == "calibrate":
        T = 1.45 * np.arange(1, case["expiries"] + 1) / case["expiries"] * g.uniform(0.98, 1.0)
        chains = [(float(t), S0 * np.sort(np.exp(math.sqrt(t) * g.uniform(-0.35, 0.35, case["strikes"])))) for t in T]
        p = (g.uniform(0.03, 0.09), g.uniform(0.03, 0.09), g.uniform(-0.8, -0.2), g.uniform(0.8, 3.0),
             g.uniform(0.3, 0.9), 0.02, 0.0)
        trial = tuple(x * g.uniform(0.97, 1.03) for x in p[:5]) + p[5:]
        return [(p, S0, chains), (trial, S0, chains)]
    strikes = np.geomspace(60.0, 160.0, case["strikes"])
    T = CHAIN if case["expiries"] == len(CHAIN) else CHAIN[:case["expiries"]]
    return [(_params("drawn", g), S0, [(t, strikes * g.uniform(0.99, 1.01)) for t in T]) for _ in range(case["sets"])]


# ------------------------------------------------------------ prepare, run

_engine = None


def _the_engine():
    global _engine   # one context per program, as the engine is meant to be used
    if _engine is None:
        _engine = Engine(0)
    return _engine


class _State:
    """What a program holds before the call; ``handle`` is a prepared batch, a server or a calibration."""

    def __init__(self, case, **kw):
        self.case, self.handle = case, None
        self.__dict__.update(kw)

    def __del__(self):
        if self.handle is not None:
            self.handle.close()


def prepare(case, seed):
    eng = _the_engine()
    if case["kind"] in ("calibrate", "swift"):
        surfaces = [(Params(*p), s, chains) for p, s, chains in _surfaces(case, seed)]
        st = _State(case, eng=eng, surfaces=surfaces)
        if case["kind"] == "calibrate":
            prm, s, chains = surfaces[0]
            st.points = [np.array([p.v0, p.theta, p.rho, p.kappa, p.sigma]) for p, _, _ in surfaces]
            st.handle = eng.calibration(s, prm.r, chains, case["trunc"])
        return st
    reqs, steps = _requests(case, seed)
    reqs = [Request(Params(*p), S0, Options(K, T, P, n), seed=sd, stream=sm) for p, K, T, P, n, sd, sm in reqs]
    cfg = Config(n_paths=case.get("paths", 1 << 14), step_mode=STEP_REFERENCE if steps else STEP_GRID,
                 steps=steps or 252, steps_per_year=STEPS_PER_YEAR, seed=reqs[0].seed,
                 precision=FP64 if case["precision"] == "fp64" else FP32, control_variate=int(case.get("cv", False)))
    st = _State(case, eng=eng, reqs=reqs, cfg=cfg)
    if case["kind"] == "graph":
        st.handle = eng.prepare_batch(reqs, cfg)
    elif case["kind"] == "serve":
        st.handle = eng.server(cfg)
    return st


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "chain":
        rq = state.reqs[0]
        price, se = state.eng.price(rq.params, rq.S0, rq.options, state.cfg)
        return {"price": price, "se": se}
    if kind == "calibrate":
        cal, (p, trial) = state.handle, state.points
        return {"price": cal.prices(p), "jacobian": cal.jacobian(p), "trial": cal.prices(trial)}
    if kind == "swift":
        out = [x for res in state.eng.swift_batch(state.surfaces, True, None, case["trunc"]) for x in res]
        return {"price": np.concatenate([p for p, _ in out]), "gradient": np.concatenate([g for _, g in out])}
    if kind == "book":
        out = state.eng.price_batch(state.reqs, state.cfg)
    elif kind == "graph":
        state.handle.launch()
        out = state.handle.collect()
    else:
        tickets = [state.handle.submit(rq) for rq in state.reqs]
        out = [state.handle.wait(t) for t in tickets]
    return {"price": np.concatenate([p for p, _ in out]), "se": np.concatenate([s for _, s in out])}


# -------------------------------------------------------------------- work

# Floating operations of a path-step: the QE step, log-spot and contracts, and two AS241 words.
_FLOPS = 110


def work(case):
    if case["kind"] in ("calibrate", "swift"):
        sets = 2 if case["kind"] == "calibrate" else case["sets"]
        J, n = 512, sets * case["expiries"]   # the usual number of frequencies of an expiry
        transforms = 2 * 5 * 2 * J * math.log2(2 * J)
        return {"flops": n * (transforms + J * (700 + case["strikes"] * 26)), "bytes": n * case["strikes"] * 7 * 8}
    if case["kind"] == "chain":
        T = _maturities(case)
        steps = case["steps"] if case["steps"] else round(STEPS_PER_YEAR * T[-1])
        if case["steps"] and len(T) > 1:   # each maturity is approached with its own width T / steps
            steps = sum(math.ceil((b - a) / (b / case["steps"])) for a, b in zip([0.0, *T], T))
        options = len(T) * case["strikes"] * (2 if case["payoffs"] == "both" else 1)
        return {"flops": case["paths"] * steps * _FLOPS + options * case["paths"] * 4, "bytes": options * 48}
    path_steps = options = folds = 0
    for T, n in _book(case):
        reach = 0
        for t in np.unique(T)[::-1]:   # paths that reach a maturity but no later one
            here = int(n[T == t].max())
            path_steps += max(0, here - reach) * round(STEPS_PER_YEAR * t)
            reach = max(reach, here)
        options += len(T)
        folds += int(n.sum())
    return {"flops": path_steps * _FLOPS + folds * 4, "bytes": options * 48}


# ------------------------------------------------------------------- exact

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_MOST_PATH_STEPS = 1.6e9   # a simulation beyond this takes too long


def exact(case, seed):
    if case["kind"] in ("calibrate", "swift"):
        out = [[_swift(p, s, t, K, case["trunc"]) for t, K in chains] for p, s, chains in _surfaces(case, seed)]
        flat = [(np.concatenate([c[0] for c in res]), np.concatenate([c[1] for c in res])) for res in out]
        if case["kind"] == "calibrate":
            return {"price": flat[0][0], "jacobian": flat[0][1], "trial": flat[1][0]}
        return {"price": np.concatenate([p for p, _ in flat]), "gradient": np.concatenate([g for _, g in flat])}
    reqs, steps = _requests(case, seed)
    plans = [_schedule(rq, steps) for rq in reqs]
    if sum(int(rq[4].max()) for rq in reqs) * max(len(p["dt"]) for p in plans) > _MOST_PATH_STEPS:
        return None
    return _simulate(reqs, plans, bool(case.get("cv", False)))


def _schedule(rq, steps):
    """The time grid: maturity j is approached with width T_j / steps_j, time adds up in doubles, and a maturity is
    priced after the first step that reaches it.  Per step its width; per maturity the step that prices it and the
    time left at that step's start."""
    T = np.unique(rq[2])
    n = [steps or max(5, int(np.rint(STEPS_PER_YEAR * t))) for t in T]
    dts, at, left = [], [], []
    t, j = 0.0, 0
    while j < len(T):
        dt = T[j] / n[j]
        tp, t = t, t + dt
        dts.append(dt)
        while j < len(T) and t >= T[j]:
            at.append(len(dts) - 1)
            left.append(T[j] - tp)
            j += 1
    after = dts[1:] + [dts[-1]]   # the width in force after a step's pricing
    return {"T": T, "n": n, "dt": np.array(dts), "after": np.array(after), "at": at, "left": left}


# SHISHUA: sixteen 64-bit state words per stream, 128 bytes per round.
_PHI = (0x9E3779B97F4A7C15, 0xF39CC0605CEDC834, 0x1082276BF3A27251, 0xF86C6A11D0C18E95, 0x2767F0B153D27B7F,
        0x0347045B5BF1827F, 0x01886F0928403002, 0xC1D64BA40F335E36, 0xF06AD7AE9717877E, 0x85839D6EFFBD7DC6,
        0x64D325D1C5371682, 0xCADD0CCCFDFFBBE1, 0x626E33B8D04B4331, 0xBBF73C790D94F79D, 0x471C4AB3ED3D82A5,
        0xFEC507705E4AE6E5)


def _shr(x, n):
    return (x >> n) & ((1 << (64 - n)) - 1)


def _i64(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _round(s, c):
    for k in range(4):
        s[4 + k] = s[4 + k] + _i64(c[k] & (2 ** 64 - 1))
        s[12 + k] = s[12 + k] + _i64(c[k] & (2 ** 64 - 1))
        c[k] += (7, 5, 3, 1)[k]
    u = [_shr(s[4 * i + k], (1, 3, 1, 3)[i]) for i in range(4) for k in range(4)]
    turn = (2, 1, 2, 1)   # lanes rotate their 32-bit elements by five or three
    t = [_shr(s[4 * i + (k + turn[i]) % 4], 32) | (s[4 * i + (k + turn[i] + 1) % 4] << 32)
         for i in range(4) for k in range(4)]
    for k in range(16):
        s[k] = t[k] + u[k]
    return ([u[k] ^ t[4 + k] for k in range(4)] + [u[8 + k] ^ t[12 + k] for k in range(4)] +
            [s[k] ^ s[12 + k] for k in range(4)] + [s[8 + k] ^ s[4 + k] for k in range(4)])


def _words(seeds, streams, blocks):
    """[blocks, 16, paths] words of the streams seeded {seed, stream, 0, 0}."""
    s = [torch.full_like(seeds, _i64(x)) for x in _PHI]
    for k in (0, 12):
        s[k] = s[k] ^ seeds
    for k in (2, 14):
        s[k] = s[k] ^ streams
    c = [0, 0, 0, 0]
    for _ in range(13):
        o = _round(s, c)
        s = [o[4 * (3 - i) + k] for i in range(4) for k in range(4)]
    out = torch.empty((blocks, 16, len(seeds)), dtype=torch.int64, device=seeds.device)
    for b in range(blocks):
        o = _round(s, c) if b else [s[4 * (3 - i) + k] for i in range(4) for k in range(4)]
        for k in range(16):
            out[b, k] = o[k]
    return out


def _uniform(w):
    """(double)w / (double)UINT64_MAX of unsigned words held as int64."""
    return (_shr(w, 32).double() * 2.0 ** 32 + (w & 0xFFFFFFFF).double()) * 2.0 ** -64


def _fma32(a, b, c):
    return (a.double() * b + c).float()


def _log32(x):
    """The inverse normal's float logarithm: reduction to [sqrt(1/2), sqrt(2)) and the odd series to s^11."""
    f32 = lambda h: float(np.float32(float.fromhex(h)))  # noqa: E731
    bits = x.view(torch.int32)
    k = (bits >> 23) - 127
    bits = (bits & 0x007FFFFF) | 0x3F800000
    up = bits > 0x3FB504F3
    m = torch.where(up, bits - 0x00800000, bits).view(torch.float32)
    kf = torch.where(up, k + 1, k).float()
    f = m - 1.0
    s = f / (2.0 + f)
    z = s * s
    p = _fma32(z, f32("0x1.745d18p-3"), f32("0x1.c71c72p-3"))
    for c in ("0x1.24924ap-2", "0x1.99999ap-2", "0x1.555556p-1"):
        p = _fma32(z, p.double(), f32(c))
    log_m = _fma32(s, (p * z).double(), (s + s).double())
    low = _fma32(kf, f32("0x1.7f7d1cp-20"), log_m.double())
    return _fma32(kf, f32("0x1.62e4p-1"), low.double())


def _poly32(c, r):
    acc = torch.full_like(r, c[0])
    for d in c[1:]:
        acc = acc * r + torch.tensor(d, dtype=torch.float32, device=r.device)
    return acc


def _normals(w):
    """AS241 (PPND16) of the words in single precision, its input stage in double."""
    P = _uniform(w)
    q = (P - 0.5).float()
    r = 0.180625 - q * q
    z = q * _poly32((2.5090809287301226727e+3, 3.3430575583588128105e+4, 6.7265770927008700853e+4,
                     4.5921953931549871457e+4, 1.3731693765509461125e+4, 1.9715909503065514427e+3,
                     1.3314166789178437745e+2, 3.3871328727963666080), r)
    z = z / _poly32((5.2264952788528545610e+3, 2.8729085735721942674e+4, 3.9307895800092710610e+4,
                     2.1213794301586595867e+4, 5.3941960214247511077e+3, 6.8718700749205790830e+2,
                     4.2313330701600911252e+1, 1.0), r)
    tail = q.abs() > np.float32(0.425)
    R = torch.where(q < 0, P, 1.0 - P).float()[tail]
    zero = R <= 0
    t = torch.sqrt(-_log32(torch.where(zero, torch.full_like(R, 0.25), R)).double()).float()
    a, b = t - 1.6, t - 5.0
    mid = _poly32((7.74545014278341407640e-4, 2.27238449892691845833e-2, 2.41780725177450611770e-1,
                   1.27045825245236838258, 3.64784832476320460504, 5.76949722146069140550,
                   4.63033784615654529590, 1.42343711074968357734), a) / _poly32(
                  (1.05075007164441684324e-9, 5.47593808499534494600e-4, 1.51986665636164571966e-2,
                   1.48103976427480074590e-1, 6.89767334985100004550e-1, 1.67638483018380384940,
                   2.05319162663775882187, 1.0), a)
    far = _poly32((2.01033439929228813265e-7, 2.71155556874348757815e-5, 1.24266094738807843860e-3,
                   2.65321895265761230930e-2, 2.96560571828504891230e-1, 1.78482653991729133580,
                   5.46378491116411436990, 6.65790464350110377720), b) / _poly32(
                  (2.04426310338993978564e-15, 1.42151175831644588870e-7, 1.84631831751005468180e-5,
                   7.86869131145613259100e-4, 1.48753612908506148525e-2, 1.36929880922735805310e-1,
                   5.99832206555887937690e-1, 1.0), b)
    v = torch.where(t <= 5.0, mid, far)
    v = torch.where(q[tail] < 0, -v, v)
    z[tail] = torch.where(zero, torch.zeros_like(v), v)
    return z


def _simulate(reqs, plans, cv):
    dev, n_sets = _DEV, len(reqs)
    f64 = dict(dtype=torch.float64, device=dev)
    n = [int(rq[4].max()) for rq in reqs]
    begin = np.concatenate([[0], np.cumsum(n)])
    P, n_steps = int(begin[-1]), max(len(p["dt"]) for p in plans)
    of = torch.repeat_interleave(torch.arange(n_sets, device=dev), torch.tensor(n, device=dev))
    k = torch.cat([torch.arange(x, device=dev) for x in n])
    seeds = (torch.tensor([rq[5] for rq in reqs], device=dev)[of] + k) & 0xFFFFFFFF
    blocks = (2 * n_steps) // 16 + 4
    words = _words(seeds, torch.tensor([rq[6] for rq in reqs], device=dev)[of], blocks)
    normals = torch.empty(words.shape, dtype=torch.float32, device=dev)
    for b in range(blocks):
        normals[b] = _normals(words[b])
    words, normals, path = words.view(-1), normals.view(-1), torch.arange(P, device=dev)

    # per step and set: the width's constants (padded with the last step's)
    rows = np.empty((n_steps, n_sets, 11))
    for r, (rq, pl) in enumerate(zip(reqs, plans)):
        v0, theta, rho, kappa, sigma, rate, q = rq[0]
        dt = np.concatenate([pl["dt"], np.full(n_steps - len(pl["dt"]), pl["dt"][-1])])
        after = np.concatenate([pl["after"], np.full(n_steps - len(pl["dt"]), pl["dt"][-1])])
        disc = np.exp(-kappa * dt)
        half = 0.5 * dt * (kappa * rho / sigma - 0.5)
        k3 = 0.5 * dt * (1.0 - rho * rho)
        rows[:, r] = np.stack([disc, sigma * sigma * disc / kappa * (1 - disc),
                               theta * sigma * sigma / (2 * kappa) * (1 - disc) ** 2,
                               -rho * kappa * theta / sigma * dt + (rate - q) * dt, half - rho / sigma,
                               half + rho / sigma, k3, k3, 0.5 * after, np.full(n_steps, theta), dt], 1)
    rows = torch.tensor(rows, **f64)

    v = torch.tensor([rq[0][0] for rq in reqs], **f64)[of]
    lx = torch.full((P,), math.log(S0), **f64)
    X = torch.full((P,), S0, **f64)
    acc, accg, y = torch.zeros(P, **f64), torch.zeros(P, **f64), torch.zeros(P, **f64)
    # the generator's two buffers: block 0 feeds the uniforms, block 1 the normals, and a buffer that runs dry
    # takes the stream's next block
    u_blk, g_blk, nxt = (torch.full((P,), x, dtype=torch.int64, device=dev) for x in (0, 1, 2))
    u_pos, g_pos = torch.zeros_like(u_blk), torch.zeros_like(u_blk)

    def take(blk, pos, nxt, need):
        dry = need & (pos == 16)
        blk = torch.where(dry, nxt, blk)
        pos = torch.where(dry, 0, pos)
        return blk, pos + need.long(), nxt + dry.long(), (blk * 16 + pos.clamp(max=15)) * P + path

    price = [np.zeros(len(rq[1])) for rq in reqs]
    se = [np.zeros(len(rq[1])) for rq in reqs]
    every = torch.ones(P, dtype=torch.bool, device=dev)
    for step in range(n_steps):
        C = rows[step, 0].tolist() if n_sets == 1 else rows[step][of].unbind(1)
        disc, cA, cB, K0, K1, K2, K3, K4, hdt, theta, _ = C
        m = (v - theta) * disc + theta
        s2 = (v * cA + cB).abs()
        psi = s2 / (m * m)
        quad = s2 < 1.5 * m * m
        g_blk, g_pos, nxt, i1 = take(g_blk, g_pos, nxt, quad)
        u_blk, u_pos, nxt, iu = take(u_blk, u_pos, nxt, ~quad)
        g_blk, g_pos, nxt, i2 = take(g_blk, g_pos, nxt, every)
        z1, U, z2 = normals[i1].double(), _uniform(words[iu]), normals[i2].double()
        inv = 2.0 / psi
        b2 = inv - 1.0 + torch.sqrt(inv * (inv - 1.0))
        a = m / (1.0 + b2)
        p = (psi - 1.0) / (psi + 1.0)
        beta = 2.0 / (m * (psi + 1.0))
        low = torch.where(p < U, torch.log((1.0 - p) / (1.0 - U)) / beta, 0.0)
        vn = torch.where(quad, a * (torch.sqrt(b2) + z1) ** 2, low)
        lx = lx + K0 + K1 * v + K2 * vn + torch.sqrt(K3 * v + K4 * vn) * z2
        v, Xp, yp, X = vn, X, y, torch.exp(lx)
        y = lx - math.log(S0)
        for r, (rq, pl) in enumerate(zip(reqs, plans)):
            lo = int(begin[r])
            for j in [j for j, at in enumerate(pl["at"]) if at == step]:
                w, T = pl["left"][j] / (pl["T"][j] / pl["n"][j]), pl["T"][j]
                sl = slice(lo, lo + n[r])
                tip = (X[sl] - Xp[sl]) * w
                asian, euro = (acc[sl] + tip) / T, Xp[sl] + tip
                geo = S0 * torch.exp((accg[sl] + (y[sl] - yp[sl]) * w) / T) if cv else None
                for i in np.nonzero(rq[2] == T)[0]:
                    price[r][i], se[r][i] = _estimate(rq, pl, i, asian, euro, geo, j)
        acc = acc + hdt * (X + Xp)
        accg = accg + hdt * (y + yp)
    return {"price": np.concatenate(price), "se": np.concatenate(se)}


def _estimate(rq, pl, i, asian, euro, geo, j):
    K, paths, disc = float(rq[1][i]), int(rq[4][i]), math.exp(-rq[0][5] * rq[2][i])
    a = ((asian if rq[3][i] == ASIAN else euro)[:paths] - K).clamp(min=0.0)
    mean, var = float(a.mean()), float(a.var(unbiased=True)) if paths > 1 else 0.0
    if geo is not None and rq[3][i] == ASIAN:
        g = (geo[:paths] - K).clamp(min=0.0)
        vg = float(g.var(unbiased=True))
        if vg > 0:
            cov = float(((a - mean) * (g - g.mean())).sum()) / (paths - 1)
            mean -= cov / vg * (float(g.mean()) - _geometric_call(rq[0], pl, j, K))
            var = max(0.0, var - cov * cov / vg)
    return disc * mean, disc * math.sqrt(var / paths)


_geo = {}   # the transform of the last (parameters, maturity), for its strikes


def _geometric_call(params, pl, j, K):
    """E[(G - K)^+] of the geometric average: a backward affine recursion over the grid for its characteristic
    function, then Lewis's integral by Gauss-Legendre."""
    key = (params, j, float(pl["T"][j]), len(pl["dt"]))
    if key not in _geo:
        _geo.clear()
        v0, theta, rho, kappa, sigma, rate, q = params
        last = pl["at"][j]
        dts, T, w = pl["dt"][:last + 1], pl["T"][j], pl["left"][j] / (pl["T"][j] / pl["n"][j])
        c = np.zeros(last + 1)
        for s in range(last):   # the trapezoid's weights on the log-spot after each step
            h = 0.5 * pl["after"][s]
            c[s] += h
            if s:
                c[s - 1] += h
        if last:
            c[last - 1] -= w
        c[last] += w
        c /= T
        C = np.cumsum(c[::-1])[::-1]
        t = np.concatenate([[0.0], np.cumsum(dts)[:-1]])
        scale = 40.0 / math.sqrt(max(1e-12, float(np.sum(C * C * (theta + (v0 - theta) * np.exp(-kappa * t)) * dts))))
        x1, w1 = np.polynomial.legendre.leggauss(256)
        x2, w2 = np.polynomial.legendre.leggauss(128)
        s = 0.5 * (x2 + 1)
        u = scale * np.concatenate([0.5 * (x1 + 1), 1 / s])
        wt = scale * np.concatenate([0.5 * w1, 0.5 * w2 / s ** 2])
        z = np.concatenate([0.5 + 1j * u, [1.0 + 0j]])
        A, b = np.zeros_like(z), np.zeros_like(z)
        for k in range(last, -1, -1):
            a, tau, s2 = z * C[k], dts[k], sigma * sigma
            beta = kappa - rho * sigma * a
            D = np.sqrt(beta * beta - s2 * a * (a - 1))
            g = (beta - D - s2 * b) / (beta + D - s2 * b)
            e = np.exp(-D * tau)
            A = A + a * (rate - q) * tau + kappa * theta / s2 * ((beta - D) * tau - 2 * np.log((1 - g * e) / (1 - g)))
            b = (beta - D - (beta + D) * g * e) / (s2 * (1 - g * e))
        phi = np.exp(A + b * v0)
        F = S0 * phi[-1].real
        _geo[key] = u, wt, phi[:-1] * np.exp(-z[:-1] * math.log(F / S0)), F
    u, wt, psi, F = _geo[key]
    return F - math.sqrt(F * K) / math.pi * float(np.sum(wt * (np.exp(1j * u * math.log(F / K)) * psi).real / (u * u + 0.25)))


def _chf(p, tau, u):
    """The characteristic function of the log-return and its derivatives in (v0, theta, rho, kappa, sigma)."""
    v0, vm, rho, kappa, sigma = p[:5]
    iu = 1j * u
    xi = kappa + sigma * rho * iu
    f = u * u - iu
    d = np.sqrt(xi * xi + sigma * sigma * f)
    sh, ch = np.sinh(d * tau / 2), np.cosh(d * tau / 2)
    A1, A2 = f * sh, d / v0 * ch + xi / v0 * sh
    A = A1 / A2
    ekt = math.exp(kappa * tau / 2)
    B = d * ekt / (v0 * A2)
    D = np.log(2 * d / (d + xi + (d - xi) * np.exp(-d * tau))) + (kappa - d) * tau / 2
    s2 = sigma * sigma
    k2 = 2 * kappa * vm / s2
    c = np.exp(kappa * vm * rho * tau * iu / sigma - A + k2 * D)
    d_rho = xi * sigma * iu / d
    A2_rho = sigma * iu * (2 + xi * tau) / (2 * d * v0) * (xi * ch + d * sh)
    B_rho = ekt / v0 * (d_rho / A2 - d / A2 ** 2 * A2_rho)
    A1_rho = iu * f * tau * xi * sigma / (2 * d) * ch
    A_rho = A1_rho / A2 - A / A2 * A2_rho
    B_kappa = -1j / (sigma * u) * B_rho + B * tau / 2
    d_sigma = (rho / sigma - 1 / xi) * d_rho + sigma * u * u / d
    A1_sigma = f * tau / 2 * d_sigma * ch
    A2_sigma = rho / sigma * A2_rho + (2 + tau * xi) / (v0 * tau * xi * iu) * A1_rho + sigma * tau * A1 / v0 / 2
    A_sigma = A1_sigma / A2 - A / A2 * A2_sigma
    t = vm * tau * iu / sigma
    return [c, -c * A / v0, c * (2 * kappa / s2 * D + kappa * rho * tau * iu / sigma),
            c * (-A_rho + k2 / d * (d_rho - d / A2 * A2_rho) + t * kappa),
            c * (-A_rho / (sigma * iu) + 2 * vm / s2 * D + k2 / B * B_kappa + t * rho),
            c * (-A_sigma - 2 * k2 / sigma * D + k2 / d * (d_sigma - d / A2 * A2_sigma) - t / sigma * rho * kappa)]


def _wavelet(p, tau, s, K, trunc):
    """The wavelet scale, range and number of frequencies of an expiry from the truncation error and the cumulants
    (whose formulas take theta and rho where their names say the volatility and the rate)."""
    m = 0
    while True:
        e = 2.0 ** m
        m += 1
        u = np.array([e * math.pi, -e * math.pi], dtype=complex)
        if not abs(_chf(p, tau, u)[0].sum()) / (4 * e * math.pi ** 2 * tau) > trunc:
            break
    s2, r, a, k, t = p[1], p[2], p[3], p[4], tau
    km = k - 2 * a * r
    E = lambda n: math.exp(-n * a * t)  # noqa: E731
    c2 = s2 / (8 * a ** 3) * (-k * k * E(2) + 4 * k * E(1) * km + 2 * a * t * (4 * a * a + k * k - 4 * a * k * r) +
                              k * (8 * a * r - 3 * k))
    c4 = 3 * k ** 2 * s2 / (64 * a ** 7) * (
        -3 * k ** 4 * E(4) - 8 * k ** 2 * E(3) * (2 * a * k * t * km + 4 * a ** 2 + k ** 2 - 6 * a * k * r)
        - 4 * E(2) * (4 * a ** 2 * k ** 2 * t ** 2 * km ** 2 +
                      2 * a * k * t * (k ** 3 - 16 * a ** 3 * r - 12 * a * k ** 2 * r + 4 * a ** 2 * k * (3 + 4 * r ** 2)) +
                      8 * a ** 4 - 3 * k ** 4 - 32 * a ** 3 * k * r + 8 * a * k ** 3 * r + 16 * a ** 2 * k ** 2 * r ** 2)
        - 8 * E(1) * (-2 * a ** 2 * k * t ** 2 * km ** 3 -
                      8 * a * t * (k ** 4 - 7 * a * k ** 3 * r + 4 * a ** 4 * r ** 2 - 8 * a ** 3 * k * r * (1 + r ** 2) +
                                   a ** 2 * k ** 2 * (3 + 14 * r ** 2)) -
                      9 * k ** 4 + 70 * a * k ** 3 * r + 32 * a ** 3 * k * r * (4 + 3 * r ** 2) -
                      16 * a ** 4 * (1 + 4 * r ** 2) - 4 * a ** 2 * k ** 2 * (9 + 40 * r ** 2))
        + 4 * a * t * (5 * k ** 4 - 40 * a * k ** 3 * r - 32 * a ** 3 * k * r * (3 + 2 * r ** 2) +
                       16 * a ** 4 * (1 + 4 * r ** 2) + 24 * a ** 2 * k ** 2 * (1 + 4 * r ** 2))
        - 73 * k ** 4 + 544 * a * k ** 3 * r + 128 * a ** 3 * k * r * (7 + 6 * r ** 2) - 32 * a ** 4 * (3 + 16 * r ** 2) -
        64 * a ** 2 * k ** 2 * (4 + 19 * r ** 2))
    width = abs(0.5 * p[1] * tau) + 10 * math.sqrt(abs(c2) + math.sqrt(abs(c4)))
    lower, upper = p[5] * tau + math.log(s / K.max()) - width, p[5] * tau + math.log(s / K.min()) + width
    scale = int(2.0 ** m)
    k1, k2 = math.ceil(scale * lower), math.floor(scale * upper)
    return scale, lower, upper, k1, k2, int(2.0 ** (math.ceil(math.log2(math.pi * abs(k1 - k2))) - 2))


def _swift(p, s, tau, K, trunc):
    """SWIFT prices and gradients of one expiry, its two transforms as matrix products."""
    scale, lower, upper, k1, k2, J = _wavelet(p, tau, s, K, trunc)
    odd, k = 2 * np.arange(J) + 1, np.arange(k1, k2 + 1)
    u = math.pi * odd / (2.0 * J) * scale
    H = lambda y: -1j * np.exp(-1j * u * y) * (1 / u - math.exp(y) / (1j + u))  # noqa: E731
    h = H(upper) - H(max(lower, 0.0))
    dev = dict(device=_DEV)
    turn = (torch.tensor(k, **dev)[:, None] * torch.tensor(odd, **dev)[None, :]) % (4 * J)
    angle = turn.double() * (math.pi / (2 * J))
    w = torch.complex(torch.cos(angle), torch.sin(angle))
    V = (w @ torch.tensor(h, **dev)).real * (math.sqrt(scale) / J)
    c = (V.to(w.dtype) @ w * (math.sqrt(scale) / J)).cpu().numpy()
    x = p[5] * tau + np.log(s / K)
    e = np.exp(-1j * np.outer(x, u)) * (math.exp(-p[5] * tau) * K)[:, None]
    out = [(e @ (g * c)).real for g in _chf(p, tau, u.astype(complex))]
    return out[0], np.stack(out[1:], axis=1)
