"""The MSE interpreter against the prediction launches of the same programs:
the two are different instantiations (operator profile, general or direct
operand paths, datapoints per thread), so each dispatch code, tile remainder
and span-group count of the MSE kernel is checked against predictions that
went another way.

Tolerance, derived: both sides square the same FP32 residual (bit-identical
predictions) and sum the squares in FP64, N <= 1.1e5 terms of relative error
2^-53 each in any order (below 2^-35), then round once to FP32: at most one
unit in the last place apart."""
import numpy as np
import pytest

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import opcodes as op

pytestmark = pytest.mark.gpu

V = 3


def _forms():
    """Every binary operator of the protected set with each kind and side of
    operand (variable, constant, spilled subtree), every unary one on a leaf
    and on a subtree, single leaves, constants only, invalid predictions."""
    x = lambda i: ([-1], [float(i)])  # noqa: E731
    c = lambda v: ([0], [v])  # noqa: E731

    def un(o, a):
        return [o] + a[0], [0.0] + a[1]

    def bi(o, a, b):
        return [o] + a[0] + b[0], [0.0] + a[1] + b[1]

    s1 = bi(op.ADD, x(0), un(op.SIN, x(1)))
    s2 = bi(op.MUL, x(2), un(op.COS, x(0)))
    es = [x(0), x(2), c(1.5), x(7), bi(op.SUB, c(2.0), c(0.5))]
    for o in op.WORKLOAD_BINARY:
        for a in (x(0), c(0.75), s1):
            for b in (x(1), c(-1.25), s2):
                es.append(bi(o, a, b))
    for o in op.WORKLOAD_UNARY:
        es += [un(o, x(1)), un(o, c(2.0)), un(o, s1)]
    deep = s1
    for k in range(6):  # needs several spill slots
        deep = bi(op.SUB if k % 2 else op.ADD, bi(op.MUL, s1, s2) if k == 0 else deep,
                  bi(op.LOOSE_DIV, deep, s2))
        if len(deep[0]) > 400:
            break
    es.append(deep)
    big = un(op.EXP_CLAMP, bi(op.MUL, c(40.0), x(0)))
    es.append(bi(op.SUB, bi(op.MUL, big, big), bi(op.MUL, big, big)))  # inf - inf: NaN rows
    es.append(bi(op.MUL, big, c(3e4)))  # finite predictions, infinite squares
    return sg.Population.from_lists(es)


def _data(n, seed):
    r = np.random.default_rng(seed)
    X = r.uniform(-3.0, 3.0, (V + 1, n)).astype(np.float32)
    X[0, : min(n, 5)] = [0.0, -0.0, 1e-10, 40000.0, -2.5][: min(n, 5)]
    return X


def _from_predictions(pred, y):
    with np.errstate(all="ignore"):
        d = (pred - y[None, :]).astype(np.float32)
        sq = (d * d).astype(np.float32).astype(np.float64)
    ok = np.isfinite(pred)
    n = ok.sum(axis=1)
    s = np.where(ok, sq, 0.0).sum(axis=1)
    with np.errstate(all="ignore"):
        return np.where(n > 0, s / n, np.nan).astype(np.float32)


def _agree(a, b):
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(np.isinf(a), np.isinf(b))
    f = np.isfinite(a)
    ulp = np.abs(a[f].view(np.int32).astype(np.int64) - b[f].view(np.int32).astype(np.int64))
    assert ulp.max(initial=0) <= 1


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1023, 1025, 8191, 33_001, 110_007])
@pytest.mark.parametrize("opts", [{}, {"smem_spill_slots": 0}, {"smem_spill_slots": 1},
                                  {"dpt": 4, "warps_per_block": 16},
                                  {"dpt": 16, "warps_per_block": 8}])
def test_mse_is_the_mean_of_the_predictions_squares(n, opts):
    pop = _forms()
    X = _data(n, n)
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X)
        want = _from_predictions(ev.predictions(pop), X[V])
    with sg.Evaluator(device=0, **opts) as ev:
        ev.set_data(X)
        _agree(ev.eval_mse(pop), want)
        s, cnt = ev.read_sums()
        with np.errstate(all="ignore"):
            _agree(np.where(cnt > 0, s / cnt, np.nan).astype(np.float32), want)
        _agree(ev.eval_mse(pop, cache=True, clear_cache=True), want)
        _agree(ev.eval_grad(pop)[0], want)


def _hard_quotients(r):
    """(a, b) whose quotient lies r / (b 2^24) (a >= b) or r / (b 2^25) (a < b)
    from the middle between two floats, for every odd 24-bit b: a 2^24 = r
    (mod b) by halving r 24 (25) times modulo b."""
    b = np.arange((1 << 23) + 1, 1 << 24, 2, dtype=np.int64)
    x = np.full(b.shape, r, np.int64) % b
    out = []
    for k in range(25):
        x = np.where(x % 2 == 0, x // 2, (x + b) // 2)
        if k == 23:
            a = x + b
            ok = a < (1 << 24)
            out.append((a[ok], b[ok]))
    ok = (x >= (1 << 23)) & (x < b)
    out.append((x[ok], b[ok]))
    return (np.concatenate([o[0] for o in out]).astype(np.float32),
            np.concatenate([o[1] for o in out]).astype(np.float32))


def _zero_error(exprs, X, n_valid=None):
    """Every prediction equals the target bit for bit: the sum of squares is 0
    over all datapoints."""
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X)
        mse = ev.eval_mse(sg.Population.from_lists(exprs))
        s, n = ev.read_sums()
    assert np.all(n == (X.shape[1] if n_valid is None else n_valid))
    assert np.all(s == 0.0) and np.all(mse == 0.0)


_DIV = [([op.LOOSE_DIV, -1, -1], [0.0, 0.0, 1.0]),
        # the accumulator as the divisor and as the dividend, products that are exact
        ([op.LOOSE_DIV, -1, op.MUL, -1, 0], [0.0, 0.0, 0.0, 1.0, 1.0]),
        ([op.LOOSE_DIV, op.MUL, -1, 0, -1], [0.0, 0.0, 0.0, 1.0, 1.0])]


@pytest.mark.parametrize("r", [1, -1, 3, -5])
def test_division_rounds_correctly_next_to_the_midpoints(r):
    a, b = _hard_quotients(r)
    assert a.size > 1_000_000
    _zero_error(_DIV, np.stack([a, b, a / b]))


@pytest.mark.parametrize("lo,hi", [(-60, 60), (-126, 127), (-149, 20), (-61, -59), (59, 61)])
def test_division_rounds_correctly_over_its_range(lo, hi):
    rng = np.random.default_rng(abs(hi))
    n = 1_500_001
    with np.errstate(all="ignore"):
        a, b = (np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi + 1, n)).astype(np.float32)
                * rng.choice([-1, 1], n).astype(np.float32) for _ in range(2))
        a[::1001] = 0.0
        b[::1013] = -0.0
        d = np.where(np.abs(b) <= np.float32(1e-9),
                     np.where(b < 0, np.float32(-1e-9), np.float32(1e-9)), b).astype(np.float32)
        y = a / d
    keep = np.isfinite(y) & (np.abs(y) < 1e19)
    a, b, y = a[keep], b[keep], y[keep]
    _zero_error(_DIV, np.stack([a, b, y]))


@pytest.mark.parametrize("case", ["mantissas", "range"])
def test_square_root_rounds_correctly(case):
    if case == "mantissas":  # every one, both parities of the exponent
        x = np.arange(0x3F800000, 0x40800000, dtype=np.uint32).view(np.float32)
    else:
        rng = np.random.default_rng(3)
        x = rng.integers(0, 0x7F800000, 3_000_001, dtype=np.int64).astype(np.uint32).view(np.float32)
        x[:4] = [0.0, 1e-45, 1.17549435e-38, 3.4e38]
    x = x * np.where(np.arange(x.size) % 3 == 0, np.float32(-1), np.float32(1))
    _zero_error([([op.LOOSE_SQRT, -1], [0.0, 0.0])], np.stack([x, np.sqrt(np.abs(x))]))


def test_protected_log_is_the_same_in_every_path():
    """log|x| of the MSE launch against the prediction launch's (scalar form)."""
    rng = np.random.default_rng(4)
    x = rng.integers(0, 0x7F800000, 4_000_003, dtype=np.int64).astype(np.uint32).view(np.float32)
    x[:6] = [0.0, -0.0, 1e-45, 1.17549435e-38, 1.1754942e-38, 3.4028235e38]
    x[1::2] *= -1
    pop = sg.Population.from_lists([([op.LOOSE_LOG, -1], [0.0, 0.0])])
    with sg.Evaluator(device=0) as ev:
        ev.set_data(np.stack([x, x]))
        y = ev.predictions(pop)[0]
    _zero_error([([op.LOOSE_LOG, -1], [0.0, 0.0])], np.stack([x, y]))


def test_reciprocals_of_the_gradient_round_correctly():
    """d/dc of c / (k x) at c = x = 1, y = 0, one datapoint: the FP32 product of
    the seed 2 / k and the partial 1 / k, both of which are correctly rounded."""
    rng = np.random.default_rng(6)
    n = 60_000
    k = np.ldexp(rng.uniform(1, 2, n), rng.integers(-62, 63, n)).astype(np.float32)
    k[:2000] = (0x3FFFFFFF - np.arange(2000)).astype(np.uint32).view(np.float32)  # just below 2
    k[2000:4000] = (0x3F800000 + np.arange(2000)).astype(np.uint32).view(np.float32)
    k = k[np.abs(k) > 1e-9]
    pop = sg.Population.from_lists([([op.LOOSE_DIV, 0, op.MUL, 0, -1], [0.0, 1.0, 0.0, float(v), 0.0])
                                    for v in k])
    with sg.Evaluator(device=0) as ev:
        ev.set_data(np.array([[1.0], [0.0]], np.float32))
        _, grad = ev.eval_grad(pop)
    r = np.float32(1) / k
    assert np.array_equal(grad[::2], (np.float32(2) * r) * r)
