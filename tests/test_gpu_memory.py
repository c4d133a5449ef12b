"""The derived rows of shared work are an option: where memory is short, calls
that need none of it come first (allocation failures are injected on the host,
sr_inject_allocation_failure)."""
import numpy as np
import pytest

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import _lib, synth
from symbolic_regression_gpu_b200.evolution import DeviceEvolution, evolve_options

pytestmark = pytest.mark.gpu

N = 120_007


@pytest.fixture(scope="module")
def work():
    w = synth.batched_workload(seed=5, E=3600, N=N)
    assert w.population.num_tokens * (N - 60_000) >= 3e9  # large enough to be shared
    with sg.Evaluator(device=0) as ev:
        ev.set_data(w.X)
        want = ev.eval_mse(w.population)
        assert ev.stats.kernel_launches == 3  # the rows', the expressions', their sums
        small = w.population.slice(0, 64)
        return w, want, small, ev.eval_mse(small)


def _ulp(a, b):
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    f = np.isfinite(b)
    return np.abs(a[f].view(np.int32).astype(np.int64) - b[f].view(np.int32).astype(np.int64)).max()


def _failing(n, call):
    assert _lib.lib.sr_inject_allocation_failure(n) == _lib.SR_OK
    try:
        return call()
    finally:
        _lib.lib.sr_inject_allocation_failure(0)


def test_an_evaluation_that_fits_without_rows_is_made(work):
    """Every allocation of the call fails in turn.  The two before the rows'
    own (the results) fail the call; any other only the rows."""
    w, want, _, _ = work
    failed = 0
    for n in range(1, 60):
        with sg.Evaluator(device=0) as ev:
            ev.set_data(w.X)
            try:
                got = _failing(n, lambda: ev.eval_mse(w.population))
            except sg.SrError as e:
                assert e.status == _lib.SR_ERR_OUT_OF_MEMORY
                failed += 1
                continue
            launches = ev.stats.kernel_launches
            assert _ulp(got, want) <= 1  # sums grouped by other spans at most
            if launches == 3:  # no allocation left to fail
                break
    else:
        pytest.fail("the call never completed with its rows")
    assert failed == 2 and n > 6


@pytest.mark.parametrize("call", ["data", "small", "cached", "grad", "adam", "predictions",
                                  "device"])
def test_calls_take_the_rows_memory_when_theirs_is_missing(work, call):
    w, _, small, small_mse = work
    with sg.Evaluator(device=0, cache_capacity=32) as ev:
        ev.set_data(w.X)
        ev.eval_mse(w.population)
        assert ev.stats.kernel_launches == 3
        if call == "data":
            _failing(1, lambda: ev.set_data(np.concatenate([w.X, w.X, w.X], axis=1)))
            ev.set_data(w.X)
        elif call == "small":
            small = sg.Population.from_lists(list(w.population) * 2)
            small_mse = np.tile(ev.eval_mse(w.population), 2)
            assert _ulp(_failing(1, lambda: ev.eval_mse(small)), small_mse) <= 1
        elif call == "cached":
            got = _failing(1, lambda: ev.eval_mse(small, cache=True))
            assert _ulp(got, small_mse) <= 1
        elif call == "grad":
            _failing(1, lambda: ev.eval_grad(small))
        elif call == "adam":
            _failing(1, lambda: ev.optimize_constants(small, steps=1))
        elif call == "predictions":
            _failing(1, lambda: ev.predictions(small, 0, 16))
        else:
            de = DeviceEvolution(ev, 64, evolve_options(w.num_vars, seed=5), stride=64)
            de.init()
            _failing(1, de.evaluate)
            assert np.isfinite(de.fitness()).any()
        if call != "small":
            assert np.array_equal(ev.eval_mse(small), small_mse, equal_nan=True)
