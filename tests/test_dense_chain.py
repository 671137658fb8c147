"""Small dense layers that follow one another, and a softmax behind them, in one launch (kernels/dense_chain.cu): the executor's way
of running such steps, which the plan lists one by one, with a line that says which are launched together."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, Graph, UnaryOp, shape


def rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def layers(widths, softmax, bias=True, seed=0, probe=None):
    r = rng(seed)
    g = Graph()
    y = x = g.input(shape(BATCH, widths[0]))
    weights = []
    for i, (k, n) in enumerate(zip(widths, widths[1:])):
        w, b = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32), r.standard_normal((1, n)).astype(np.float32)
        weights.append((w, b if bias else np.zeros((1, n), np.float32)))
        y = g.linear(y, g.constant_tensor(w))
        if bias:
            y = g.add(y, g.constant_tensor(b))
        if i + 2 < len(widths):
            y = g.relu(y)
        if probe == i:
            g.output(g.unary(UnaryOp.TANH, y))
    g.output(g.softmax(y, 1) if softmax else y)
    return g, weights


def want(x, weights, softmax):
    y = x.astype(np.float64)
    for i, (w, b) in enumerate(weights):
        y = y @ w.T.astype(np.float64) + b
        if i + 1 < len(weights):
            y = np.maximum(y, 0)
    if softmax:
        y = np.exp(y - y.max(1, keepdims=True))
        y /= y.sum(1, keepdims=True)
    return y


def together(g, rows, mode=MATH_F32):
    """(first, last) of the steps that are launched together"""
    lines = [l.split(":")[0].split(" ")[1].split("..") for l in plan_describe(g, rows, mode).splitlines() if l.startswith("together")]
    return [(int(a), int(b)) for a, b in lines]


def test_runs():
    def runs(widths, softmax, rows=8, **more):
        return together(layers(widths, softmax, **more)[0], rows)
    assert runs([16, 32, 32, 4], True) == [(0, 3)] and runs([16, 32, 32, 4], False) == [(0, 2)] and runs([256, 3], True) == [(0, 1)]
    assert runs([256, 3], False) == [] and runs([300, 3], True) == [] and runs([20, 129, 3], False) == []      # one layer; too long; too wide
    assert runs([8] * 7, True) == [(0, 3), (4, 6)]                                                             # four layers at most
    assert runs([64, 64, 64, 8], True) == [(1, 3)]                                                             # weights of 7424 floats
    assert runs([64, 64, 8], True, 500) and runs([96, 64], True) and not runs([96, 64], True, 2000)
    g = layers([64, 64, 8], True)[0]                                                                           # on tensor cores from 64 rows on
    assert together(g, 63, MATH_TF32) and together(g, 500, MATH_TF32) and together(g, 1500, MATH_TF32) == [(1, 2)]
    assert not together(layers([96, 64], True)[0], 64, MATH_TF32)
    assert together(layers([16, 32, 32, 4], True)[0], 65536, MATH_TF32) == [(0, 3)]
    assert runs([16, 32, 32, 4], True, probe=1) == [(0, 1), (3, 4)]                                            # a result that is read elsewhere


CASES = [  # widths of the layers, softmax, bias
    ([16, 32, 32, 4], True, True), ([256, 3], True, True), ([5, 9, 8, 1], False, True), ([1, 96, 33], True, False), ([7, 31, 64, 8, 2], True, True),
    ([20, 8, 40], False, True), ([33, 100], True, True),
]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 7, 64, 2369])
@pytest.mark.parametrize("widths,softmax,bias", CASES)
@pytest.mark.parametrize("mode", [MATH_F32, MATH_TF32])
def test_values(rows, widths, softmax, bias, mode):
    from kyanite_b200.executor import CudaExecutor
    g, weights = layers(widths, softmax, bias, seed=len(widths))
    x = rng(rows).standard_normal((rows, widths[0])).astype(np.float32)
    expected = want(x, weights, softmax)
    with CudaExecutor(0, g, rows, math_mode=mode) as ex:
        got, = ex.evaluate([x])
        # a few layers of f32 sums of at most 256 terms; steps that stay by themselves may round their operands to 11 bits
        rounded = "/tc" in "".join(l for i, l in enumerate(plan_describe(g, rows, mode).splitlines()[1:]) if not any(a <= i <= b for a, b in together(g, rows, mode)))
        assert np.abs(got - expected).max() <= (4e-3 if rounded else 4e-6) * np.abs(expected).max()
        steps, launches = ex.step_count()
        assert launches == steps - sum(last - first for first, last in together(g, rows, mode))
        ex.set_profile(True)                       # (the same launches, timed)
        np.testing.assert_array_equal(got, ex.evaluate([x])[0])
        profile = [l for l in ex.last_profile().splitlines() if not l.startswith("total")]
        assert len(profile) == steps and sum("launched with" in l for l in profile) == sum(last - first + 1 for first, last in together(g, rows, mode))
        ex.set_profile(False)
        np.testing.assert_array_equal(got, ex.evaluate([x])[0])


@pytest.mark.gpu
def test_a_result_that_is_read_elsewhere_is_stored():
    from kyanite_b200.executor import CudaExecutor
    g, weights = layers([16, 32, 32, 4], True, probe=1)
    x = rng(1).standard_normal((9, 16)).astype(np.float32)
    with CudaExecutor(0, g, 9, math_mode=MATH_F32) as ex:
        hidden, got = ex.evaluate([x])
    h = np.tanh(np.maximum(want(x, weights[:2], False), 0))
    assert np.abs(hidden - h).max() <= 4e-6 and np.abs(got - want(x, weights, True)).max() <= 4e-6


@pytest.mark.gpu
@pytest.mark.parametrize("widths", [[7, 9, 30, 3], [5, 33, 12], [8, 11, 6, 21]])
@pytest.mark.parametrize("rows", [3, 2369])
def test_infinities_stay_infinities(widths, rows):
    """Positive weights and no activation: a row with an infinity is infinite in every column, behind layers of any width."""
    from kyanite_b200.executor import CudaExecutor
    g = Graph()
    y = g.input(shape(BATCH, widths[0]))
    for k, n in zip(widths, widths[1:]):
        y = g.linear(y, g.constant_tensor(np.full((n, k), 0.25, np.float32)))
    g.output(y)
    x = np.ones((rows, widths[0]), np.float32)
    x[1, 0], x[2, 3] = np.inf, -np.inf
    with CudaExecutor(0, g, rows, math_mode=MATH_F32) as ex:
        got, = ex.evaluate([x])
    assert (got[1] == np.inf).all() and (got[2] == -np.inf).all() and np.isfinite(np.delete(got, [1, 2], 0)).all()
