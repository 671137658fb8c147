"""Softmax over rows that are not 16-byte aligned and layer norms of few long rows, at the edges of their variants, against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, CudaExecutor
from kyanite_b200.graph import Graph, shape
from oracle.cpu_eval import cpu_eval_graph

pytestmark = pytest.mark.gpu


def check(g, inputs, scale):
    with CudaExecutor(0, g, 0, math_mode=MATH_F32) as ex:
        got, = ex.evaluate(inputs)
    expected, = cpu_eval_graph(g.to_bytes(), 0, inputs)
    # f32 exponentials and roots (2 ulp), sums of up to 2^16 terms in another order: 1e-5 of the largest value
    assert np.abs(got.astype(np.float64) - expected).max() <= 1e-5 * max(scale, np.abs(expected).max())


@pytest.mark.parametrize("length", [1025, 2047, 2049, 4097, 5913, 8191, 8193])
@pytest.mark.parametrize("term", [False, True])
def test_softmax(length, term):
    rng = np.random.default_rng(length)
    g = Graph()
    x = g.mul(g.input(shape(3, length)), g.scalar(1.5))
    if term:
        x = g.add(x, g.broadcast(g.input(shape(1, length)), shape(3, length)))
    g.output(g.softmax(x, 1))
    inputs = [rng.standard_normal((3, length)).astype(np.float32)] + ([rng.standard_normal((1, length)).astype(np.float32)] if term else [])
    inputs[0][1, 7] = -np.inf
    check(g, inputs, 0.0)


# eight CTAs a row up to 74 rows, one from 75 on; two and three float4 a thread; a slice that ends early
@pytest.mark.parametrize("rows,length", [(1, 8196), (2, 24576), (2, 24580), (3, 32768), (74, 32772), (75, 32772), (32, 40960), (3, 49152)])
@pytest.mark.parametrize("residual", [False, True])
def test_layernorm(rows, length, residual):
    rng = np.random.default_rng(length + rows)
    g = Graph()
    x = g.input(shape(rows, length))
    if residual:
        x = g.add(x, g.input(shape(rows, length)))
    g.output(g.layernorm(x, 1, 1e-5))
    check(g, [(rng.standard_normal((rows, length)) + 3).astype(np.float32) for _ in range(1 + residual)], 1.0)
