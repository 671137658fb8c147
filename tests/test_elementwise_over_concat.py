"""An elementwise expression over a concatenation is computed part by part (a step per part, no copy).  The reference copies
every part and runs the expression on the result: kn-cuda-eval/src/planner.rs:835-923."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, DType, Graph, SliceRange, UnaryOp, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph


def rotary(dtype, rows, heads, d):
    g = Graph()
    r = np.random.Generator(np.random.PCG64(1))
    t = g.input(shape(BATCH, rows, heads, d), dtype)
    cos, sin = (g.constant_tensor(r.standard_normal((1, rows, 1, d)).astype(dtype.np)) for _ in range(2))
    lo, hi = g.slice(t, 3, SliceRange(0, d // 2)), g.slice(t, 3, SliceRange(d // 2, d))
    rotated = g.concat([g.unary(UnaryOp.NEG, hi), lo], 3)
    g.output(g.add(g.mul(t, cos), g.mul(rotated, sin)))
    return g


def joined(axis, sizes, read_twice=False):
    """(concat of a, |b|, a constant) * x - x"""
    g = Graph()
    r = np.random.Generator(np.random.PCG64(2))
    full = [3, 5, 4]
    full[axis] = sum(sizes)
    part = lambda n: [n if i == axis else full[i] for i in range(3)]  # noqa: E731
    a, b = g.input(shape(*part(sizes[0]))), g.input(shape(*part(sizes[1])))
    c = g.constant_tensor(r.standard_normal(part(sizes[2])).astype(np.float32))
    x = g.input(shape(*full))
    j = g.concat([a, g.unary(UnaryOp.ABS, b), c], axis)
    g.output(g.sub(g.mul(j, x), x))
    if read_twice:
        g.output(j)
    return g


def elementwise_steps(g, batch):
    return [l for l in plan_describe(g, batch, MATH_TF32).splitlines() if l.startswith("step") and " Scalar " in l]


def test_steps():
    assert len(elementwise_steps(rotary(DType.F16, 7, 2, 64), 2)) == 2
    assert len(elementwise_steps(joined(1, [1, 6, 2]), 0)) == 3
    assert any("copy" in l for l in elementwise_steps(joined(1, [1, 6, 2], read_twice=True), 0))   # it is needed as it is


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [lambda: rotary(DType.F16, 7, 2, 64), lambda: rotary(DType.F32, 7, 2, 64), lambda: rotary(DType.F16, 5, 3, 20),
                                   lambda: joined(0, [1, 6, 2]), lambda: joined(1, [3, 1, 4]), lambda: joined(2, [4, 4, 8]),
                                   lambda: joined(2, [1, 2, 3], read_twice=True)])
def test_matches_oracle(graph):
    from kyanite_b200.executor import CudaExecutor
    g = graph()
    r = np.random.Generator(np.random.PCG64(3))
    inputs = [r.standard_normal([d.eval(2) for d in g[v].shape]).astype(g[v].dtype.np) for v in g.inputs]
    expected = cpu_eval_graph(g.to_bytes(), 2, inputs)
    with CudaExecutor(0, g, 2, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)
    # three operations, each rounded once (a multiply-add may round once less): two units of the storage type
    tol = 2e-3 if any(e.dtype == np.float16 for e in expected) else 1e-6
    assert_tensors_match(expected, got, tol, tol, abs_scaled=True)
