"""Gradients of a few large trees among many small ones: the sums per span of a
gradient mode are laid out for the expressions it evaluates, not for the
population.

Results: each tree's are those of a population of the few alone.  The same
spans are added in the same order, so errors are equal bit for bit; gradients
too in forward mode, and in reverse mode (FP64 atomics in any order, fewer than
1e5 of them a constant, 1e5 x 2^-53 of the terms' scale) to 1e-6 after the
rounding to 32 bits, the targets being far enough off that no gradient cancels
below 1e-3 of its terms."""
import numpy as np
import pytest
import torch

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import opcodes as op

pytestmark = pytest.mark.gpu

V, N, E = 3, 400_000, 20_000


def _sum_of(k, rng):
    """sum over k terms of c x: k constants, 4k - 1 tokens."""
    t, v = [], []
    for i in range(k):
        if i + 1 < k:
            t.append(op.ADD)
            v.append(0.0)
        t += [op.MUL, 0, -1]
        v += [0.0, float(rng.uniform(0.5, 2.0)), float(rng.integers(V))]
    return t, v


@pytest.mark.parametrize("constants", [6, 12])
def test_a_few_trees_among_many(constants):
    rng = np.random.default_rng(constants)
    few = [_sum_of(constants, rng) for _ in range(5)]
    many = [_sum_of(1 + i % 2, rng) for i in range(E)]
    place = [7, 1000, 9999, 15_000, E + 4]
    mixed = list(many)
    for at, tree in zip(place, few):
        mixed.insert(at, tree)
    few, mixed = sg.Population.from_lists(few), sg.Population.from_lists(mixed)
    X = rng.uniform(1.0, 5.0, (V + 1, N)).astype(np.float32)
    X[V] = -50.0
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X[:, :512])
        ev.eval_grad(mixed)  # loads every kernel
        ev.set_data(X)
        want_mse, want_grad = ev.eval_grad(few)
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X)
        before = torch.cuda.mem_get_info()[0]
        mse, grad = ev.eval_grad(mixed)
        used = before - torch.cuda.mem_get_info()[0]
    # Programs, constants, results and the sums of the many: tens of MB; sums of
    # the few for every expression of the population: 0.6 GB (reverse mode) and more.
    assert used < 256 << 20
    assert np.array_equal(mse[place], want_mse)
    first = np.concatenate([[0], np.cumsum([sum(k == 0 for k in t) for t, _ in mixed])])
    got = np.concatenate([grad[first[i]:first[i + 1]] for i in place])
    assert got.shape == want_grad.shape
    if constants <= 8:
        assert np.array_equal(got, want_grad)
    else:
        assert np.allclose(got, want_grad, rtol=1e-6, atol=0.0)
