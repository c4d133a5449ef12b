"""What a call says it evaluated (node_evals_executed, the declared operator
counts) is what it evaluates: equal expressions, shared subtrees and subtrees of
constants count once, or not at all where the device folds them."""
import numpy as np
import pytest

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import opcodes as op
from symbolic_regression_gpu_b200 import synth
from symbolic_regression_gpu_b200.evolution import DeviceEvolution, evolve_options

pytestmark = pytest.mark.gpu

# (2 * 3) + x0: five tokens, three of them left once the product is a constant;
# sin(x1); 1.5: nothing to fold.
FOLDED = [([op.ADD, op.MUL, 0, 0, -1], [0.0, 0.0, 2.0, 3.0, 0.0]),
          ([op.SIN, -1], [0.0, 1.0]), ([0], [1.5])]


@pytest.mark.parametrize("call", ["plain", "batched", "cached", "grad", "device"])
def test_folded_constants(call):
    N = 1000
    pop = sg.Population.from_lists(FOLDED)
    X = np.random.default_rng(1).uniform(-1.0, 1.0, (3, N)).astype(np.float32)
    with sg.Evaluator(device=0, cache_capacity=8) as ev:
        ev.set_data(X)
        if call == "grad":
            ev.eval_grad(pop)
        elif call == "device":
            de = DeviceEvolution(ev, 3, evolve_options(2, seed=1), stride=8)
            de.load(pop)
            de.evaluate()
            de.fitness()
        else:
            ev.eval_mse(pop, cache=call == "cached", plain=call == "plain")
        st = ev.stats
    assert st.node_evals == 8 * N
    # The plain kernel and small batched launches evaluate everything.
    assert st.node_evals_executed == (8 if call in ("plain", "batched") else 6) * N


def test_shared_work_counts_once():
    N = 150_007
    rng = np.random.default_rng(2)
    gen = synth.TreeGen(rng, 4)
    trees = [gen.sized_tree(int(n)) for n in rng.integers(10, 40, 40)]
    one = sg.Population.from_lists(trees)
    many = sg.Population.from_lists(trees * 60)
    assert many.num_tokens * (N - 60_000) >= 3e9 > one.num_tokens * (N - 60_000)
    X = rng.uniform(-3.0, 3.0, (5, N)).astype(np.float32)
    with sg.Evaluator(device=0) as ev:
        ev.set_data(X)
        ev.eval_mse(one)
        alone = type(ev.stats).from_buffer_copy(ev.stats)
        ev.eval_mse(many)
        st = ev.stats
    assert alone.node_evals == alone.node_evals_executed == one.num_tokens * N
    assert st.node_evals == 60 * alone.node_evals
    # The distinct programs, their shared subtrees a leaf each, and up to 24 of
    # those subtrees (at most 64 tokens).
    assert 0 < st.node_evals_executed <= alone.node_evals + 24 * 64 * N
    assert 0 < st.declared_sfu_ops <= alone.declared_sfu_ops
    assert 0 < st.declared_fp32_ops <= alone.declared_fp32_ops
