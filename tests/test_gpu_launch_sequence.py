"""Work counters between launch sequences: whatever ran, was captured or failed
before, a sequence hands out every work item.

The results are the ones of an undisturbed evaluation, bit for bit (one launch
shape, one order of additions).  Before each attempt another data set is
evaluated in the same shape, so that a work item left out shows."""
import numpy as np
import pytest
import torch

import symbolic_regression_gpu_b200 as sg
from symbolic_regression_gpu_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def work():
    w = synth.plain_workload(seed=3, E=512, N=65_536)
    with _evaluator() as ev:
        ev.set_data(w.X)
        want = ev.eval_mse(w.population)
        assert ev.stats.work_items > 2 * ev.stats.blocks  # items beyond each block's first
    return w, want


def _evaluator(**kw):
    return sg.Evaluator(device=0, dpt=8, warps_per_block=8, **kw)


def _dirty(ev, w):
    """Other results in the span sums, then used-up counters."""
    ev.set_data(w.X[:, ::-1] + 1.0)
    ev.eval_mse(w.population)
    ev.set_data(w.X)
    ev.predictions(w.population)


@pytest.mark.parametrize("retry", ["graph", "one-shot"])
def test_a_failed_graph_instantiation_leaves_the_next_launch_whole(work, retry):
    w, want = work
    with _evaluator(use_graphs=True) as ev:
        _dirty(ev, w)
        ev.prepare(w.population)
        assert _lib.lib.sr_inject_allocation_failure(1) == _lib.SR_OK
        try:
            with pytest.raises(sg.SrError) as e:
                ev.launch()
        finally:
            _lib.lib.sr_inject_allocation_failure(0)
        assert e.value.status == _lib.SR_ERR_OUT_OF_MEMORY
        if retry == "graph":
            ev.launch()
            got = ev.read_mse()
            ev.launch()
            assert np.array_equal(ev.read_mse(), got, equal_nan=True)
        else:
            got = ev.eval_mse(w.population)
    assert np.array_equal(got, want, equal_nan=True)


def test_a_launch_captured_by_the_stream_s_owner(work):
    w, want = work
    stream = torch.cuda.Stream()
    with _evaluator(stream=stream) as ev:
        _dirty(ev, w)
        ev.prepare(w.population)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            ev.launch()
        ev.launch()  # nothing captured has run yet
        assert np.array_equal(ev.read_mse(), want, equal_nan=True)
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
            stream.synchronize()
            assert np.array_equal(ev.read_mse(), want, equal_nan=True)
        del graph
