"""The persistent matmul with one and with two groups of epilogue warps: short and longer sums, with and without a bias and an
activation, tiles with row and column tails, against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, CudaExecutor, plan_describe
from kyanite_b200.graph import DType, Graph, UnaryOp, shape
from oracle.cpu_eval import cpu_eval_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 64, 256, 260, 512, 520])   # (f32 without a bias: one group)
@pytest.mark.parametrize("kind", ["f32", "bias", "gelu", "f16"])
def test_values(k, kind):
    half = kind == "f16"
    b, m, n = (40, 300, 520) if kind in ("f32", "f16") else (1, 12000, 520)   # more than one round of tiles
    rng = np.random.default_rng(k)
    g = Graph()
    x = g.input(shape(b, m, k), DType.F16 if half else DType.F32)
    w = (rng.standard_normal((b, k, n)) / np.sqrt(k)).astype(np.float16 if half else np.float32)
    y = g.batched_mat_mul(x, g.constant_tensor(w))
    if kind in ("bias", "gelu"):
        y = g.add(y, g.constant_tensor(rng.standard_normal((1, 1, n)).astype(np.float32)))
    if kind == "gelu":   # x / 2 * (1 + erf(x / sqrt 2))
        y = g.mul(g.mul(y, g.scalar(0.5)), g.add(g.unary(UnaryOp.ERF, g.mul(y, g.scalar(float(np.sqrt(0.5))))), g.scalar(1.0)))
    g.output(y)
    line, = [l for l in plan_describe(g, 0, MATH_TF32).splitlines() if l.startswith("step") and " matmul " in l]
    assert " Gemm/tc " in line and "splitk" not in line      # (more than a round of tiles, no slices: the persistent kernel)
    a = rng.standard_normal((b, m, k)).astype(np.float16 if half else np.float32)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate([a])
    expected, = cpu_eval_graph(g.to_bytes(), 0, [a])
    # sums of k products of about unit variance together, less than 8 of it: operands rounded to 2^-12 each (TF32; two of them, the
    # errors of k products add up as their root); f16 results are both rounded, so sums an f32 rounding apart may land on neighbours,
    # which lie 2^-8 apart from 4 to 8; GELU's slope is at most 1.13
    bound = 2.0 ** -8 if half else 6 * 2 * 2.0 ** -12 * 1.13
    assert np.abs(got.astype(np.float64) - expected.astype(np.float64)).max() <= bound
