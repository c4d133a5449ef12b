"""Shared work under launch shapes given from outside, tuned ones, and programs
of more spill slots than the derived rows were counted for: the results of the
same expressions evaluated a few at a time, where nothing is shared.

Tolerance, derived: every operator gets the same operands on both sides; the
sums differ by their grouping alone (double-doubles over spans, FP64 within a
lane's tiles), so the FP32 results are at most one unit in the last place apart."""
import numpy as np
import pytest

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import opcodes as op
from symbolic_regression_gpu_b200 import synth

pytestmark = pytest.mark.gpu

N = 120_007


def _balanced(rng, depth, V):
    """A tree that spills depth - 1 values, unlike any other."""
    if depth == 0:
        if rng.random() < 0.5:
            return [-1], [float(rng.integers(V))]
        return [0], [float(rng.uniform(-2.0, 2.0))]
    a, b = _balanced(rng, depth - 1, V), _balanced(rng, depth - 1, V)
    o = int(rng.choice([op.ADD, op.SUB, op.MUL]))
    if depth == 1:  # not constants only
        a = [-1], [float(rng.integers(V))]
    return [o] + a[0] + b[0], [0.0] + a[1] + b[1]


def _population(V, depth):
    rng = np.random.default_rng(100 * V + depth)
    gen = synth.TreeGen(rng, V)
    base = [gen.sized_tree(int(n)) for n in rng.integers(5, 40, 600)]
    out = list(base)
    while len(out) < 2600:
        out.append(synth.crossover(rng, base[int(rng.integers(len(base)))],
                                   base[int(rng.integers(len(base)))], 120))
    out += [_balanced(rng, depth, V) for _ in range(3)]
    return sg.Population.from_lists(out)


_CACHE = {}


def _case(V, depth):
    if (V, depth) not in _CACHE:
        pop = _population(V, depth)
        assert pop.num_tokens * (N - 60_000) >= 3e9  # large enough to be shared
        X = np.random.default_rng(V).uniform(-3.0, 3.0, (V + 1, N)).astype(np.float32)
        want = []
        with sg.Evaluator(device=0) as ev:
            ev.set_data(X)
            for a in range(0, pop.num_exprs, 400):
                part = pop.slice(a, min(a + 400, pop.num_exprs))
                assert part.num_tokens * (N - 60_000) < 3e9
                want.append(ev.eval_mse(part))
        _CACHE[V, depth] = pop, X, np.concatenate(want)
    return _CACHE[V, depth]


def _agree(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    f = np.isfinite(want)
    ulp = np.abs(got[f].view(np.int32).astype(np.int64) - want[f].view(np.int32).astype(np.int64))
    assert ulp.max() <= 1


# Launches: the derived rows', the expressions', the combination of their sums.
@pytest.mark.parametrize("V,depth,opts,launches", [
    (5, 4, {}, 3),                       # three spill slots
    (5, 6, {}, 3),                       # five: compiled again with fewer rows
    (12, 6, {}, 3),
    (20, 6, {}, 2),                      # no room for four rows: none
    (5, 6, {"autotune": True}, 3),
    (5, 6, {"dpt": 4, "warps_per_block": 16}, 3),
    (5, 7, {"smem_spill_slots": 0}, 3),
    # Shapes whose spill slots leave the rows no shared memory.
    (5, 7, {"smem_spill_slots": 16}, 2),
    (5, 7, {"dpt": 16, "warps_per_block": 16, "smem_spill_slots": 16}, 2),
])
def test_shapes_that_meet_shared_work(V, depth, opts, launches):
    pop, X, want = _case(V, depth)
    with sg.Evaluator(device=0, **opts) as ev:
        ev.set_data(X)
        got = ev.eval_mse(pop)
        assert ev.stats.kernel_launches == launches
        again = ev.eval_mse(pop)
    _agree(got, want)
    assert np.array_equal(again, got, equal_nan=True)
