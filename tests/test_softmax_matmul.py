"""softmax(c * x + term) . V in f32 as one step, at the edges of its row tiles, key blocks and column panels, against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, MATH_TF32, CudaExecutor, plan_describe
from kyanite_b200.graph import Graph, shape
from oracle.cpu_eval import cpu_eval_graph


def graph(b, m, n, dv, term=None, heads=0, split=False):
    g = Graph()
    x = g.mul(g.input(shape(b, m, n)), g.scalar(0.7))
    if term == "input":
        x = g.add(x, g.broadcast(g.input(shape(1, 1, n)), shape(b, m, n)))
    elif term == "causal":
        x = g.add(x, g.broadcast(g.constant_tensor(np.triu(np.full((1, m, n), -np.inf, np.float32), 1)), shape(b, m, n)))
    if split:   # V as a head split of [B * keys, heads * dv]
        v = g.view(g.permute(g.view(g.input(shape(b // heads * n, heads * dv)), shape(b // heads, n, heads, dv)), [0, 2, 1, 3]), shape(b, n, dv))
    else:
        v = g.input(shape(b, n, dv))
    y = g.batched_mat_mul(g.softmax(x, 2), v)
    if heads:
        y = g.view(g.permute(g.view(y, shape(b // heads, heads, m, dv)), [0, 2, 1, 3]), shape(b // heads * m, heads * dv))
    g.output(y)
    return g


def steps(g, mode):
    return [line for line in plan_describe(g, 0, mode).splitlines() if line.startswith("step")]


def test_route():
    assert len(steps(graph(12, 120, 77, 64), MATH_TF32)) == 1
    assert len(steps(graph(12, 60, 60, 64, "input", heads=6, split=True), MATH_TF32)) == 1
    assert len(steps(graph(3, 20, 30, 6), MATH_TF32)) > 1          # columns that are no whole 16-byte pieces
    assert len(steps(graph(3, 20, 1025, 8), MATH_TF32)) > 1        # rows too long to keep
    assert len(steps(graph(3, 20, 128, 8), MATH_TF32)) == 1 and len(steps(graph(3, 20, 129, 8), MATH_TF32)) == 2
    assert "softmax(x)" not in plan_describe(graph(64, 512, 512, 64), 0, MATH_TF32)   # for the tensor cores
    assert len(steps(graph(12, 120, 77, 64), MATH_F32)) == 2


def test_transposed_head_split_is_read_in_place():
    g = Graph()
    split = g.view(g.permute(g.view(g.input(shape(200, 128)), shape(2, 100, 4, 32)), [0, 2, 1, 3]), shape(8, 100, 32))
    g.output(g.batched_mat_mul(g.softmax(g.input(shape(8, 70, 32)), 2), g.permute(split, [0, 2, 1])))
    plan = steps(g, MATH_TF32)
    assert len(plan) == 2 and "Softmax" in plan[0] and "read in place: operand b" in plan[1], plan


CASES = [(1, 1, 1, 4, None, 0, False), (2, 15, 127, 40, "input", 0, False), (2, 17, 129, 64, None, 0, False), (3, 33, 33, 68, "causal", 0, False),
         (4, 16, 1024, 128, None, 2, False), (8, 1000, 77, 80, None, 8, True), (40, 130, 200, 36, "input", 0, False), (6, 50, 300, 24, "input", 3, True),
         (5, 31, 125, 128, "input", 0, False), (40, 130, 126, 100, None, 8, True), (4, 9, 128, 88, None, 4, True), (2, 5, 5, 72, "causal", 0, False), (12, 120, 120, 64, None, 12, True), (2, 130, 257, 80, None, 1, False)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_against_oracle(case):
    g = graph(*case)
    rng = np.random.default_rng(sum(case[:4]))
    inputs = [rng.standard_normal([d.eval(0) for d in g[v].shape]).astype(np.float32) * 2 for v in g.inputs]
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate(inputs)
    expected, = cpu_eval_graph(g.to_bytes(), 0, inputs)
    # f32 exponentials (2 ulp) and f32 sums of at most 1024 terms in another order
    assert np.abs(got.astype(np.float64) - expected).max() <= 1e-5 * np.abs(expected).max()


@pytest.mark.gpu
def test_masked_rows_and_values_that_are_not_finite():
    """A row of -infinity is NaN, an infinite value behind a probability of zero too, as with the three operations one by one."""
    g = graph(2, 20, 40, 8)
    rng = np.random.default_rng(3)
    x, v = rng.standard_normal((2, 20, 40)).astype(np.float32), rng.standard_normal((2, 40, 8)).astype(np.float32)
    x[0, 3] = -np.inf
    x[1, :5, 7] = -np.inf
    v[1, 7, 2] = np.inf
    v[0, 11, 5] = np.nan
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate([x, v])
    with np.errstate(all="ignore"):
        expected, = cpu_eval_graph(g.to_bytes(), 0, [x, v])
    np.testing.assert_array_equal(np.isnan(got), np.isnan(expected))
    np.testing.assert_allclose(got, expected, rtol=1e-4, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,split", [(1, 2, False), (16, 40, False), (20, 300, True), (2600, 77, False)])
def test_values_near_the_end_of_the_range(m, n, split):
    """The probabilities are divided by their sum before the product: a weighted mean is no larger than the largest value."""
    b, dv, heads = 2, 8, 2
    g = graph(b, m, n, dv, None, heads if split else 0, split)
    rng = np.random.default_rng(m + n)
    x = np.zeros((b, m, n), np.float32)
    v = (rng.uniform(2e38, 3e38, (b, n, dv)) * np.where(np.arange(dv) < 4, 1.0, rng.choice([-1.0, 1.0], (b, n, dv)))).astype(np.float32)
    operand = v.transpose(1, 0, 2).reshape(n, heads * dv) if split else v
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate([x, operand])
    expected = np.broadcast_to(v.astype(np.float64).mean(axis=1, keepdims=True), (b, m, dv))
    if split:
        expected = expected.transpose(1, 0, 2).reshape(m, heads * dv)
    # equal probabilities, rounded once, and f32 sums of at most 300 terms: 300 * 2^-24 of the terms' mean size
    np.testing.assert_allclose(got, expected, rtol=0, atol=300 * 2.0 ** -24 * 3e38)


@pytest.mark.gpu
@pytest.mark.parametrize("b,m,n,dv", [(12, 4, 128, 64), (4, 1, 77, 128), (12, 120, 120, 64), (12, 1, 1024, 32), (4, 33, 700, 88)])
def test_error_against_64_bits(b, m, n, dv):
    """Of a term: exponential 2 ulp at most (half an ulp on average), division and product half an ulp each, and some ten additions on
    its way into the sum, whose errors are independent; the scores' own rounding (of up to 6) is 2^-22 at most: 3.6 units of 2^-24
    in all.  (One running sum over 256 of 1024 keys is 5.8 units off.)"""
    g = graph(b, m, n, dv)
    rng = np.random.default_rng(n)
    x, v = rng.standard_normal((b, m, n)).astype(np.float32) * 2, rng.standard_normal((b, n, dv)).astype(np.float32)
    s = x.astype(np.float64) * 0.7
    e = np.exp(s - s.max(axis=2, keepdims=True))
    expected = e / e.sum(axis=2, keepdims=True) @ v.astype(np.float64)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate([x, v])
    assert np.linalg.norm(got - expected) <= 3.6 * 2.0 ** -24 * np.linalg.norm(expected)
