"""Layer norms of rows of up to 1024 elements, at the edges of the rules that give a row a warp, 128 or 256 threads, with deviations
from tiny to too large for the quotient without branches, against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, CudaExecutor
from kyanite_b200.graph import Graph, shape
from oracle.cpu_eval import cpu_eval_graph


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 296, 297, 1776, 1777])
@pytest.mark.parametrize("length", [256, 260, 512, 516, 768, 1022, 1024, 1028])
@pytest.mark.parametrize("residual", [False, True])
def test_layernorm(rows, length, residual):
    rng = np.random.default_rng(length + rows)
    g = Graph()
    x = g.input(shape(rows, length))
    if residual:
        x = g.add(x, g.input(shape(rows, length)))
    g.output(g.layernorm(x, 1, 1e-5))
    inputs = [(rng.standard_normal((rows, length)) + 3).astype(np.float32) for _ in range(1 + residual)]
    for a in inputs:   # rows of other scales: deviations far below the root of epsilon, and past 1e15
        for row, scale in ((1, 1e-12), (2, 1e17), (3, 0.0), (4, 1e6)):
            if row < rows:
                a[row] *= np.float32(scale)
    with CudaExecutor(0, g, 0, math_mode=MATH_F32) as ex:
        got, = ex.evaluate(inputs)
    expected, = cpu_eval_graph(g.to_bytes(), 0, inputs)
    # f32 roots and quotients (2 ulp), sums of up to 1028 terms in another order: 1e-5 of a row's largest value
    assert (np.abs(got.astype(np.float64) - expected) <= 1e-5 * np.maximum(np.abs(expected).max(axis=1, keepdims=True), 1e-30)).all()
