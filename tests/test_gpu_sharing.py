"""Shared work of large launches (equal expressions, folded constants, derived
rows) against the same expressions evaluated a few at a time, where nothing is
shared: the same results.

Tolerance, derived: every operator gets the same operands on both sides, so
predictions are bit-identical; the sums differ by their span grouping alone
(double-doubles), so the FP32 results are at most one unit in the last place
apart."""
import numpy as np
import pytest

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import opcodes as op
from symbolic_regression_gpu_b200 import synth

pytestmark = pytest.mark.gpu


def _population(seed, E, V, every):
    rng = np.random.default_rng(seed)
    binary = op.BINARY_OPS if every else op.WORKLOAD_BINARY
    unary = op.UNARY_OPS if every else op.WORKLOAD_UNARY
    gen = synth.TreeGen(rng, V, binary=binary, unary=unary)
    base = [gen.sized_tree(int(n)) for n in rng.integers(1, 40, E // 4)]
    out = list(base)
    while len(out) < E:
        k = int(rng.integers(3))
        a = base[int(rng.integers(len(base)))]
        if k == 0:
            out.append(a)  # an equal expression
        elif k == 1:
            out.append(synth.crossover(rng, a, base[int(rng.integers(len(base)))], 120))
        else:
            out.append(synth.mutate(gen, a, 120))
    c = lambda v: ([0], [v])  # noqa: E731

    def bi(o, a, b):
        return [o] + a[0] + b[0], [0.0] + a[1] + b[1]

    for o in binary:  # constants only: folded whole, signs of zero and infinities among them
        for a in (0.0, -0.0, 1e-10, -2.5, 3e38):
            out.append(bi(o, c(a), c(-0.75)))
            out.append(bi(o, ([-1], [0.0]), bi(o, c(1.25), c(a))))
    for o in unary:
        for a in (0.0, -0.0, 0.3, -2.5, 90.0, 40000.0):
            out.append(([o, 0], [0.0, a]))
    out.append(([-1], [float(V)]))      # not a variable: 0
    out.append(bi(op.ADD, ([-1], [-3.0]), ([-1], [0.0])))
    big = bi(op.ADD, c(1.0), c(2.0))
    for _ in range(40):                 # more constants than one folded subtree holds
        big = bi(op.MUL, big, c(1.01))
    out.append(bi(op.ADD, big, ([-1], [0.0])))
    return sg.Population.from_lists(out)


@pytest.mark.parametrize("every", [False, True])
@pytest.mark.parametrize("V,N", [(1, 140_007), (5, 170_001), (12, 141_000), (20, 139_011)])
def test_shared_work_changes_no_result(V, N, every):
    pop = _population(3 * V + every, 2400, V, every)
    assert pop.num_tokens * (N - 60_000) >= 3e9  # large enough to be shared
    rng = np.random.default_rng(V)
    X = rng.uniform(-3.0, 3.0, (V + 1, N)).astype(np.float32)
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X)
        got = ev.eval_mse(pop)
        s, n = ev.read_sums()
        again = ev.eval_mse(pop)
        ev.prepare(pop)
        ev.launch()
        ev.launch()
        launched = ev.read_mse()
        parts = []
        step = 500
        for a in range(0, pop.num_exprs, step):
            part = pop.slice(a, min(a + step, pop.num_exprs))
            assert part.num_tokens * (N - 60_000) < 3e9
            parts.append(ev.eval_mse(part))
    with sg.Evaluator(device=0, use_graphs=True) as ev:
        ev.set_data(X)
        ev.prepare(pop)
        ev.launch()
        ev.launch()
        graphed = ev.read_mse()
    want = np.concatenate(parts)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    f = np.isfinite(want)
    ulp = np.abs(got[f].view(np.int32).astype(np.int64) - want[f].view(np.int32).astype(np.int64))
    assert ulp.max() <= 1
    with np.errstate(all="ignore"):
        assert np.array_equal(np.where(n > 0, s / n, np.nan).astype(np.float32), got, equal_nan=True)
    for other in (again, launched, graphed):
        assert np.array_equal(other, got, equal_nan=True)


def test_device_populations_fold_constants_to_the_same_values():
    """The device compiler evaluates subtrees of constants; the host's small
    launches evaluate them at every datapoint."""
    from symbolic_regression_gpu_b200.evolution import DeviceEvolution, evolve_options

    V, N = 3, 5003
    pop = _population(77, 800, V, True)
    keep = [i for i in range(pop.num_exprs) if pop.offsets[i + 1] - pop.offsets[i] <= 120]
    pop = pop.subset(keep)
    X = np.random.default_rng(7).uniform(-3.0, 3.0, (V + 1, N)).astype(np.float32)
    assert N < 60_000  # nothing shared on the host's side
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X)
        want = ev.eval_mse(pop)
        de = DeviceEvolution(ev, pop.num_exprs, evolve_options(V, seed=1), stride=130)
        de.load(pop)
        de.evaluate()
        got = de.fitness()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    f = np.isfinite(want)
    ulp = np.abs(got[f].view(np.int32).astype(np.int64) - want[f].view(np.int32).astype(np.int64))
    assert ulp.max() <= 1
