"""An elementwise expression over a concatenation is computed part by part (a step per part, no copy).  The reference copies
every part and runs the expression on the result: kn-cuda-eval/src/planner.rs:835-923."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, BinaryOp, DType, Graph, ReduceOp, SliceRange, UnaryOp, shape
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


def joined(axis, sizes, read_twice=False, dtype=DType.F32):
    """(concat of a, |b|, a constant) * x - x"""
    g = Graph()
    r = np.random.Generator(np.random.PCG64(2))
    full = [3, 5, 4]
    full[axis] = sum(sizes)
    part = lambda n: [n if i == axis else full[i] for i in range(3)]  # noqa: E731
    a, b = g.input(shape(*part(sizes[0])), dtype), g.input(shape(*part(sizes[1])), dtype)
    c = g.constant_tensor(r.standard_normal(part(sizes[2])).astype(dtype.np))
    x = g.input(shape(*full), dtype)
    j = g.concat([a, g.unary(UnaryOp.ABS, b), c], axis)
    g.output(g.sub(g.mul(j, x), x))
    if read_twice:
        g.output(j)
    return g


def normalised_part(dtype):
    """concat of (the root-mean-square norm of x, y), times z"""
    g = Graph()
    x, y, z = g.input(shape(64, 256), dtype), g.input(shape(64, 256), dtype), g.input(shape(64, 512), dtype)
    t = g.value_cast(x, DType.F32) if dtype == DType.F16 else x
    mean = g.view(g.reduce(g.pow(t, g.scalar(2.0)), [1], ReduceOp.MEAN), shape(64, 1))
    n = g.mul(g.binary(BinaryOp.DIV, t, g.unary(UnaryOp.SQRT, g.add(mean, g.scalar(1e-5)))), g.constant_tensor(np.ones((1, 256), np.float32)))
    g.output(g.mul(g.concat([g.value_cast(n, dtype) if dtype == DType.F16 else n, y], 1), z))
    return g


def elementwise_steps(g, batch):
    return [l for l in plan_describe(g, batch, MATH_TF32).splitlines() if l.startswith("step") and " Scalar " in l]


def test_steps():
    assert len(elementwise_steps(rotary(DType.F16, 7, 2, 64), 2)) == 2
    assert len(elementwise_steps(joined(1, [1, 6, 2]), 0)) == 3
    assert any("copy" in l for l in elementwise_steps(joined(1, [1, 6, 2], read_twice=True), 0))   # it is needed as it is
    for dtype, kinds in ((DType.F32, "f32->f32"), (DType.F16, "f16->f16")):
        steps = [l for l in plan_describe(normalised_part(dtype), 0, MATH_TF32).splitlines() if l.startswith("step")]
        assert len(steps) == 3 and "rmsnorm" in steps[0] and kinds in steps[0], steps     # (not taken apart into its operations)


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [lambda: rotary(DType.F16, 7, 2, 64), lambda: rotary(DType.F32, 7, 2, 64), lambda: rotary(DType.F16, 5, 3, 20),
                                   lambda: joined(0, [1, 6, 2]), lambda: joined(1, [3, 1, 4]), lambda: joined(2, [4, 4, 8]),
                                   lambda: joined(2, [1, 2, 3], read_twice=True),
                                   # f16 parts that start off 16 bytes, of whole and of odd numbers of 16-byte pieces
                                   lambda: joined(2, [3, 16, 13], dtype=DType.F16), lambda: joined(2, [8, 5, 3], dtype=DType.F16),
                                   lambda: joined(1, [3, 1, 4], dtype=DType.F16), lambda: normalised_part(DType.F32),
                                   lambda: normalised_part(DType.F16)])
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
