"""What this framework is measured on: calls of its public entry points over
the range of sizes its users have.

Every case is one pass of one entry point (population fitness, subtree-cached
fitness, device-resident fitness, gradients of the constants, constant
optimisation, predictions) on a population and a dataset drawn from a seed.
The populations have the shapes of the repository's own configurations
(``symbolic_regression_gpu_b200.synth``): ramped half-and-half trees, trees
bred by 20 generations of subtree crossover and mutation, children of a few
parents, trees with a given number of constants, long trees, and the device
generator's random trees over every operator.  The generators are restated
here on ``random.Random`` because a case is prepared many times.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from symbolic_regression_gpu_b200 import Evaluator, Population, opcodes as op
from symbolic_regression_gpu_b200.evolution import DeviceEvolution, evolve_options


# ---- the cases ----------------------------------------------------------------

def listed():
    return [
        # One call on a handful of candidates over a small table: an
        # interactive check, a unit of a larger search.  Latency is all of it.
        dict(name="fit tiny", kind="fit", trees="ramped", E=64, N=4096, V=3, lo=1.0, hi=5.0),
        # A generation of a small search on a measured data set (a thousand
        # rows, none of the sizes a power of two).
        dict(name="fit small", kind="fit", trees="bred", E=500, N=1000, V=2, lo=-3.0, hi=3.0),
        # The plain configuration: 1,000 ramped half-and-half trees x 100,000.
        dict(name="fit plain", kind="fit", trees="ramped", E=1000, N=100_000, V=3, lo=1.0, hi=5.0),
        # A generation of ragged sizes: an odd population, an odd data set.
        dict(name="fit ragged", kind="fit", trees="bred", E=1531, N=250_007, V=7, lo=-3.0, hi=3.0),
        # The batched configuration (the headline): 10,000 bred trees x 1M.
        dict(name="fit batched", kind="fit", trees="bred", E=10_000, N=1_000_000, V=5, lo=-3.0,
             hi=3.0),
        # The large configuration's trees and data set (3-127 tokens, 10
        # variables, 4M datapoints), a slice of its population.
        dict(name="fit long", kind="fit", trees="long", E=8000, N=4_000_000, V=10, lo=-5.0, hi=5.0),
        # The cache configuration: children of 256 parents, through the
        # subtree cache, each call a new generation's (the cache is cleared).
        dict(name="fit cached", kind="cached", trees="shared", E=4096, N=1_000_000, V=9, lo=0.5,
             hi=10.0),
        # A generation of the device loop: a device-resident population over
        # every operator, compiled and evaluated there, fitness read back.
        dict(name="fit device", kind="device", trees="random", E=2000, N=100_000, V=3, lo=1.0,
             hi=5.0),
        # The constant-gradient configuration: 4,096 trees with 1-8 constants.
        dict(name="grad few", kind="grad", trees="consts", E=4096, N=262_144, V=4, lo=1.0, hi=5.0,
             cmin=1, cmax=8),
        # Trees with more constants than forward mode takes (reverse mode).
        dict(name="grad many", kind="grad", trees="consts", E=512, N=65_536, V=4, lo=1.0, hi=5.0,
             cmin=9, cmax=24),
        # Constant optimisation inside a search: a few Adam steps on the
        # candidates of one generation, an odd data set.
        dict(name="adam", kind="adam", trees="consts", E=1000, N=20_001, V=4, lo=1.0, hi=5.0,
             cmin=1, cmax=8, steps=10),
        # Predictions of the best candidates on the whole data set.
        dict(name="predict", kind="predict", trees="ramped", E=50, N=100_000, V=3, lo=1.0, hi=5.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones
    as they fall, any variable count, the work bounded by the listed cases'."""
    kind = rng.choice(["fit", "fit", "fit", "fit", "cached", "device", "grad", "grad", "adam",
                       "predict"])
    lo, hi = rng.choice([(1.0, 5.0), (-3.0, 3.0), (0.5, 10.0), (-5.0, 5.0)])
    c = dict(kind=kind, V=rng.randint(1, 12), lo=lo, hi=hi)
    most = dict(fit=2e9, cached=1e9, device=2e8, grad=5e8, adam=2e7, predict=5e6)[kind]
    if kind == "fit":
        c["trees"] = rng.choice(["ramped", "bred", "bred", "long"])
    elif kind == "cached":
        c["trees"] = "shared"
    elif kind == "device":
        c["trees"] = "random"
    elif kind == "predict":
        c["trees"] = "ramped"
    else:
        c["trees"] = "consts"
        c["cmin"], c["cmax"] = rng.choice([(1, 4), (1, 8), (3, 16)])
        if kind == "adam":
            c["steps"] = rng.randint(3, 20)
    c["E"] = _log_int(rng, 8, 200) if kind == "predict" else _log_int(rng, 32, 5000)
    c["N"] = _log_int(rng, 500, min(2_000_000, max(1000.0, most / c["E"])))
    return c


# ---- populations ----------------------------------------------------------------

class _Trees:
    """Random prefix trees (token list, value list) over the workload operators
    or, with ``every``, over all of them."""

    def __init__(self, rng, V, p_const=0.3, every=False):
        self.rng, self.V, self.p_const, self.p_unary = rng, V, p_const, 0.35
        self.binary = op.BINARY_OPS if every else op.WORKLOAD_BINARY
        self.unary = op.UNARY_OPS if every else op.WORKLOAD_UNARY

    def leaf(self, t, v):
        if self.rng.random() < self.p_const:
            t.append(0)
            v.append(float(np.float32(self.rng.uniform(-5.0, 5.0))))
        else:
            t.append(-1)
            v.append(float(self.rng.randrange(self.V)))

    def depth(self, d, full, t, v):
        r = self.rng.random
        if d <= 0 or (not full and r() < 0.3):
            self.leaf(t, v)
            return t, v
        unary = r() < self.p_unary
        t.append(self.rng.choice(self.unary if unary else self.binary))
        v.append(0.0)
        self.depth(d - 1, full, t, v)
        if not unary:
            self.depth(d - 1, full, t, v)
        return t, v

    def sized(self, size, t, v):
        if size <= 1:
            self.leaf(t, v)
        elif size == 2 or (size > 3 and self.rng.random() < self.p_unary * 0.6):
            t.append(self.rng.choice(self.unary))
            v.append(0.0)
            self.sized(size - 1, t, v)
        else:
            t.append(self.rng.choice(self.binary))
            v.append(0.0)
            left = self.rng.randrange(1, size - 1)
            self.sized(left, t, v)
            self.sized(size - 1 - left, t, v)
        return t, v

    def length(self, lo, hi, mean):
        p = 1.0 / (mean - lo + 1.0)
        while True:
            n = lo + int(math.log(1.0 - self.rng.random()) / math.log(1.0 - p))
            if n <= hi:
                return n


def _sizes(t):
    n = len(t)
    s = [1] * n
    for i in range(n - 1, -1, -1):
        k = t[i]
        if k > 0:
            a = s[i + 1]
            s[i] = 1 + a + s[i + 1 + a] if k < 10 else 1 + a
    return s


def _mutated(g, e, most, least):
    t, v, s = e
    i = g.rng.randrange(len(t))
    room = most - (len(t) - s[i])
    lo, hi = max(1, s[i] - 2), min(room, s[i] + 2)
    nt, nv = g.sized(g.rng.randint(lo, max(lo, hi)), [], [])
    ct = t[:i] + nt + t[i + s[i]:]
    if len(ct) < least or len(ct) > most:
        return e
    return ct, v[:i] + nv + v[i + s[i]:], _sizes(ct)


def _crossed(rng, a, b, most, least):
    (ta, va, sa), (tb, vb, sb) = a, b
    i = rng.randrange(len(ta))
    n = sa[i]
    for _ in range(min(len(tb), 32)):
        j = rng.randrange(len(tb))
        m = sb[j]
        if n // 2 <= m <= 2 * n + 1 and least <= len(ta) - n + m <= most:
            t = ta[:i] + tb[j:j + m] + ta[i + n:]
            return t, va[:i] + vb[j:j + m] + va[i + n:], _sizes(t)
    return a


def _bred(g, E, generations=20):
    rng = g.rng
    pop = []
    for _ in range(E):
        t, v = g.sized(g.length(3, 63, 15.0), [], [])
        pop.append((t, v, _sizes(t)))
    for _ in range(generations):
        nxt = rng.sample(pop, max(1, E // 20))
        while len(nxt) < E:
            a = pop[rng.randrange(E)]
            nxt.append(_mutated(g, a, 63, 3) if rng.random() < 0.35 else
                       _crossed(rng, a, pop[rng.randrange(E)], 63, 3))
        pop = nxt
    return pop


def _shared(g, E, parents=256, pool_size=48):
    rng = g.rng
    pool = []
    while len(pool) < pool_size:
        t, v = g.depth(rng.randint(2, 4), rng.random() < 0.5, [], [])
        if len(t) >= 3:
            pool.append((t, v, _sizes(t)))

    def plant(e):
        t, v, s = e
        i = rng.randrange(len(t))
        p = rng.choice(pool)
        ct = t[:i] + p[0] + t[i + s[i]:]
        return ct, v[:i] + p[1] + v[i + s[i]:], _sizes(ct)

    par = []
    for _ in range(parents):
        t, v = g.depth(rng.randint(3, 5), False, [], [])
        e = (t, v, _sizes(t))
        for _ in range(rng.randint(1, 2)):
            e = plant(e)
        par.append(e)
    out = []
    for _ in range(E):
        a, r = rng.choice(par), rng.random()
        if r < 0.5:
            e = _crossed(rng, a, rng.choice(par), 63, 3)
        elif r < 0.8:
            e = _mutated(g, a, 63, 3)
        else:
            e = plant(a)
        out.append(e if 3 <= len(e[0]) <= 63 else a)
    return out


def _with_constants(g, draw, want):
    """A tree of draw() with room for `want` constants, its leaves turned into
    constants, or back into variables, until it has that many."""
    rng = g.rng
    while True:
        t, v = draw()
        cs = [i for i, k in enumerate(t) if k == 0]
        xs = [i for i, k in enumerate(t) if k == -1]
        if len(cs) + len(xs) >= want:
            break
    rng.shuffle(cs)
    rng.shuffle(xs)
    for i in cs[want:]:
        t[i], v[i] = -1, float(rng.randrange(g.V))
    for i in xs[:max(0, want - len(cs))]:
        t[i], v[i] = 0, float(np.float32(rng.uniform(-5.0, 5.0)))
    return t, v


def _population(case, seed):
    rng = random.Random(1_000_003 * seed + 17)
    E, V, kind = case["E"], case["V"], case["trees"]
    g = _Trees(rng, V, p_const=0.35 if kind == "consts" else 0.3, every=kind == "random")
    if kind == "ramped":
        es = [g.depth(2 + (i // 2) % 5, i % 2 == 0, [], []) for i in range(E)]
    elif kind == "bred":
        es = _bred(g, E)
    elif kind == "long":
        es = [_with_constants(g, lambda: g.sized(g.length(3, 127, 25.0), [], []),
                              rng.randint(0, 8)) for _ in range(E)]
    elif kind == "shared":
        es = _shared(g, E)
    elif kind == "random":
        es = [g.sized(g.length(3, 60, 14.0), [], []) for _ in range(E)]
    else:
        lo = 5 if case["cmax"] <= 8 else 2 * case["cmin"] + 1
        hi = 63 if case["cmax"] <= 8 else 127
        # So many constants each, in turn: their total does not vary.
        few, many = case["cmin"], case["cmax"]
        es = [_with_constants(g, lambda: g.sized(g.length(lo, hi, lo + 13.0), [], []),
                              few + i % (many - few + 1)) for i in range(E)]
    off = np.zeros(E + 1, np.int64)
    np.cumsum([len(e[0]) for e in es], out=off[1:])
    return Population(np.array([k for e in es for k in e[0]], np.int32),
                      np.array([x for e in es for x in e[1]], np.float64), off)


def _dataset(case, seed):
    """[(V+1), N] float32 on the GPU: uniform variables, the target a smooth
    law of them with 1 % noise."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    V, N = case["V"], case["N"]
    X = torch.empty((V + 1, N), dtype=torch.float32, device="cuda")
    X[:V].uniform_(case["lo"], case["hi"], generator=gen)
    a, b = X[0], X[V - 1]
    X[V] = 1.5 * a * b + torch.sin(2.0 * a) - 0.5 * b
    X[V] += 0.01 * torch.randn(N, dtype=torch.float32, device="cuda", generator=gen)
    return X


# ---- a user's program ------------------------------------------------------------

class _State:
    pass


def prepare(case, seed):
    """The evaluator with its data set, and the population (on the host; the
    device loop's in device memory)."""
    s = _State()
    s.case = case
    X = _dataset(case, seed)
    torch.cuda.synchronize()
    s.ev = Evaluator()
    s.ev.set_data_device(X)
    if case["kind"] == "device":
        s.evo = DeviceEvolution(s.ev, case["E"], evolve_options(case["V"], seed=seed), stride=64)
        s.evo.load(_population(case, seed))
    else:
        s.pop = _population(case, seed)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "fit":
        return s.ev.eval_mse(s.pop)
    if kind == "cached":
        return s.ev.eval_mse(s.pop, cache=True, clear_cache=True)
    if kind == "device":
        s.evo.evaluate()
        return s.evo.fitness()
    if kind == "grad":
        return s.ev.eval_grad(s.pop)
    if kind == "adam":
        return s.ev.optimize_constants(s.pop, steps=s.case["steps"])
    return s.ev.predictions(s.pop)


def work(case):
    """Operators of the population x datapoints (one operation each, three for
    the squared error; a gradient's product with each operator's partial
    another two), the data set and the tokens read once, results written."""
    E, N, V = case["E"], case["N"], case["V"]
    mean = dict(ramped=14.0, bred=17.0, long=30.0, shared=16.0, random=14.0,
                consts=22.0 if case.get("cmax", 8) <= 8 else 51.0)[case["trees"]]
    ops = 0.57 * mean
    times = 1.0
    if case["kind"] in ("grad", "adam"):
        ops *= 3.0
    if case["kind"] == "adam":
        times = case["steps"] + 1.0
    flops = times * E * N * (ops + 3.0)
    rows = 4.0 * N * (V + 1)
    out = 4.0 * E * (N if case["kind"] == "predict" else 1)
    return {"bytes": rows + 12.0 * E * mean + out, "flops": flops}


# ---- the same in 64 bits -----------------------------------------------------------

def _protect(d):
    return torch.where(d.abs() <= 1e-9, torch.where(d < 0, -1e-9, 1e-9).to(d.dtype), d)


def _log_or(x):
    zero = x == 0
    return torch.where(zero, torch.full_like(x, -1e9), torch.log(torch.where(zero, 1.0, x).abs()))


def _sqrt_abs(x):
    zero = x == 0
    return torch.where(zero, torch.zeros_like(x), torch.sqrt(torch.where(zero, 1.0, x).abs()))


_OPS = {
    1: lambda a, b: a + b, 2: lambda a, b: a - b, 3: lambda a, b: a * b,
    4: lambda a, b: torch.where(b == 0, torch.nan, a / b), 5: torch.pow,
    6: torch.fmin, 7: torch.fmax, 8: lambda a, b: a / _protect(b),
    9: lambda a, b: torch.where((a == 0) & (b == 0), 0.0, torch.pow(a.abs(), b)),
    10: torch.sin, 11: torch.cos, 12: torch.tan, 13: torch.sinh, 14: torch.cosh, 15: torch.tanh,
    16: torch.exp, 17: torch.log, 18: lambda a: 1.0 / a, 19: torch.asin, 20: torch.acos,
    21: torch.atan, 22: _log_or, 23: lambda a: 1.0 / _protect(a), 24: torch.abs, 25: torch.neg,
    26: torch.sqrt, 27: _sqrt_abs, 32: lambda a: torch.exp(torch.clamp(a, max=80.0)),
}


def _evaluate(t, v, X, consts=None):
    """The expression over X's rows, in their type; constants as float32 values, or
    the given tensors in token order."""
    V = X.shape[0] - 1
    k = len(consts) if consts is not None else 0
    stack = []
    for i in range(len(t) - 1, -1, -1):
        tok = t[i]
        if tok == 0:
            if consts is not None:
                k -= 1
                stack.append(consts[k])
            else:
                stack.append(torch.full((), float(np.float32(v[i])), dtype=X.dtype,
                                        device=X.device))
        elif tok == -1:
            j = int(v[i])
            stack.append(X[j] if 0 <= j < V else torch.zeros((), dtype=X.dtype, device=X.device))
        elif tok < 10:
            a = stack.pop()
            stack.append(_OPS[tok](a, stack.pop()))
        else:
            stack.append(_OPS[tok](stack.pop()))
    return stack[0].expand(X.shape[1])


_FLT_MAX = float(np.finfo(np.float32).max)


def _squares(t, v, X, consts=None):
    """Squared errors, with the product's own overflow of 32 bits, and which
    datapoints count."""
    p = _evaluate(t, v, X, consts)
    valid = p.abs() <= _FLT_MAX
    sq = ((p - X[-1]) ** 2).double()
    return torch.where(sq > _FLT_MAX, torch.inf, sq), valid


def _mse(exprs, X):
    out = np.full(len(exprs), np.nan)
    got = []
    for t, v in exprs:
        sq, valid = _squares(t, v, X)
        n = valid.sum()
        got.append(torch.where(n > 0, torch.where(valid, sq, 0.0).sum() / n, torch.nan))
    if got:
        out[:] = torch.stack(got).cpu().numpy()
    return out


def _results(case, seed, dtype):
    X = _dataset(case, seed).to(dtype)
    exprs = [(t.tolist(), v.tolist()) for t, v in _population(case, seed)]
    if case["kind"] == "predict":
        return (np.stack([_evaluate(t, v, X).cpu().numpy() for t, v in exprs]),)
    if case["kind"] != "grad":
        return (_mse(exprs, X),)
    mse, grad = [], []
    for t, v in exprs:
        cs = [torch.full((), float(np.float32(x)), dtype=dtype, device="cuda",
                         requires_grad=True) for k, x in zip(t, v) if k == 0]
        sq, valid = _squares(t, v, X, cs)
        n = valid.sum()
        m = torch.where(valid, sq, 0.0).sum() / n
        mse.append(m.detach())
        if cs:
            g = torch.autograd.grad(m, cs, allow_unused=True)
            grad += [torch.zeros((), dtype=dtype, device="cuda") if x is None else x for x in g]
    return torch.stack(mse).cpu().numpy(), torch.stack(grad).cpu().numpy()


def exact(case, seed):
    """The outputs in 64 bits.  One whose largest entries are so
    ill-conditioned that plain 32-bit arithmetic does not come near has no
    value to compare with."""
    if case["kind"] == "adam":
        return None  # a step's direction is the sign of what may be rounding alone
    out = []
    for x, y in zip(_results(case, seed, torch.float64), _results(case, seed, torch.float32)):
        y = y.astype(np.float64)
        fine = np.isfinite(x) & np.isfinite(y)
        near = np.linalg.norm(x[fine] - y[fine]) <= 0.02 * np.linalg.norm(x[fine])
        out.append(x if near else None)
    if all(x is None for x in out):
        return None
    return out[0] if len(out) == 1 else tuple(out)
