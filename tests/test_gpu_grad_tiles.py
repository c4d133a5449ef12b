"""Gradients in both modes at the edges of tiles and of forward mode's pairs of
tiles (whose products are summed together), with 1 to 8 constants, partials that
are zero somewhere and datapoints whose residual is, against the FP32 bytecode
emulator.

Tolerance, derived: as for the larger emulator comparison, only the FP64
summation order (at most (N + 64) 2^-53 of the summed magnitudes) and the FP32 rounding
of the returned gradient (half an ulp) differ."""
import numpy as np
import pytest

from emulate import adjoint_bytecode, tangent_bytecode
from symbolic_regression_gpu_b200 import Evaluator, Population, _lib
from symbolic_regression_gpu_b200 import opcodes as op
from symbolic_regression_gpu_b200.evaluator import compile_population

pytestmark = pytest.mark.gpu


def _bi(o, a, b):
    return [o] + a[0] + b[0], [0.0] + a[1] + b[1]


def _x(v):
    return [-1], [float(v)]


def _c(v):
    return [0], [float(v)]


def _population(V):
    out = []
    for nc in range(1, 9):  # constants on either side, under products and differences
        t = _bi(op.ADD, _x(0), _c(0.5))
        for k in range(1, nc):
            o = (op.MUL, op.SUB, op.ADD, op.LOOSE_DIV)[k % 4]
            leaf = _bi(op.MUL, _x(k % V), _c(0.25 * k - 1.1))
            t = _bi(o, t, leaf) if k % 2 else _bi(o, leaf, t)
        out.append(t)
        out.append(_bi(op.MUL, _bi(op.SUB, _x(1), _x(1)), t))   # a zero partial everywhere
        out.append(_bi(op.MUL, _x(2), t))                        # zero where x2 is
        out.append(_bi(op.LOOSE_DIV, t, _x(2)))                  # the flat region
    return Population.from_lists(out)


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("N", [1, 127, 128, 129, 256, 257, 384, 641])
def test_tile_edges_match_the_emulator(N, reverse):
    V = 3
    rng = np.random.default_rng(N)
    X = rng.uniform(-2.0, 2.0, (V + 1, N)).astype(np.float32)
    X[2, ::5] = 0.0
    pop = _population(V)
    X[V, ::3] = X[0, ::3] + np.float32(0.5)  # the first expression's value: a zero residual
    mode = _lib.SR_GRAD_CHECKPOINT | (_lib.SR_GRAD_REVERSE_ONLY if reverse else 0)
    emulate = adjoint_bytecode if reverse else tangent_bytecode
    with Evaluator(device=0) as ev:
        ev.set_data(X)
        mse, g = ev.eval_grad(pop, mode=mode)
    code, offs, _ = compile_population(pop, V)
    co = pop.constant_offsets()
    for e in range(pop.num_exprs):
        nc = int(co[e + 1] - co[e])
        with np.errstate(all="ignore"):
            m_e, g_e, gabs = emulate(code[offs[e]:offs[e + 1]], X, V, nc, dtype=np.float32,
                                     with_abs=True)
        got = g[co[e]:co[e + 1]]
        assert np.array_equal(np.isfinite(got), np.isfinite(g_e))
        f = np.isfinite(g_e)
        excess = np.abs(got[f] - g_e[f]) - 2.0**-24 * np.abs(g_e[f])
        assert np.all(excess <= (N + 64) * 2.0**-53 * gabs[f] + 1e-45)
        assert np.isclose(mse[e], m_e, rtol=1e-6, equal_nan=True)
