"""Elementwise programs that are compiled (kernels/elementwise_fixed.cu): which ones are, and that they give the oracle's values at
the sizes where a thread takes more positions, in every rank, with broadcast operands along any axis."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import DType, Graph, UnaryOp, shape
from oracle.cpu_eval import cpu_eval_graph
from test_elementwise_over_concat import rotary

F16, F32 = DType.F16, DType.F32


def silu(g, x):
    return g.mul(x, g.unary(UnaryOp.SIGMOID, x))


def program(name, dtype, dims, row_shape):
    """The program over tensors of `dims`; scale and shift are of `row_shape`."""
    g = Graph()
    x = g.input(shape(*dims), dtype)
    if name == "sum":
        y = g.add(x, g.input(shape(*dims), dtype))
    elif name == "swiglu":
        y = g.mul(silu(g, x), g.input(shape(*dims), dtype))
    elif name == "geglu":
        gate = g.input(shape(*dims), dtype)
        half, root, one = (g.scalar(v, dtype) for v in (0.5, 0.70710677, 1.0))
        y = g.mul(x, g.mul(g.mul(gate, half), g.add(g.unary(UnaryOp.ERF, g.mul(gate, root)), one)))
    else:
        y = g.add(g.mul(x, g.input(shape(*row_shape), dtype)), g.input(shape(*row_shape), dtype))
        if name == "affine_silu":
            y = silu(g, y)
    g.output(y)
    return g


SHAPES = [((7, 24), (1, 24)), ((5, 3, 8), (5, 1, 1)), ((2, 3, 5, 16), (1, 3, 1, 1)), ((3, 5, 7, 8), (1, 5, 7, 8)), ((593, 2056), (593, 1)),
          ((1187, 1048), (1, 1048)), ((3, 331, 2440), (1, 331, 1)), ((2341, 2080), (1, 1))]
CASES = [(n, d, s, r) for n in ("sum", "affine", "affine_silu", "swiglu", "geglu") for d in (F32, F16) for s, r in SHAPES if (n, d) != ("geglu", F16)]


def compiled(g, batch=0):
    return [" compiled" in l for l in plan_describe(g, batch, MATH_TF32).splitlines() if l.startswith("step") and " Scalar " in l]


@pytest.mark.parametrize("name,dtype,dims,row", CASES)
def test_is_compiled(name, dtype, dims, row):
    assert compiled(program(name, dtype, dims, row)) == [True]


def test_others_are_interpreted():
    g = Graph()
    g.output(g.sub(g.input(shape(8, 8)), g.input(shape(8, 8))))
    assert compiled(g) == [False]
    assert compiled(program("sum", F32, (5, 7), None)) == [False]      # rows that are no multiple of four
    assert compiled(rotary(F16, 7, 2, 64), 2) == compiled(rotary(F32, 7, 2, 64), 2) == [True, True]


def check(g, batch, seed, exact, atol=0.0):
    from kyanite_b200.executor import CudaExecutor
    r = np.random.default_rng(seed)
    inputs = [r.standard_normal([d.eval(batch) for d in g[v].shape]).astype(g[v].dtype.np) for v in g.inputs]
    for x in inputs:
        if x.size >= 24:
            x.flat[np.linspace(0, x.size - 1, 5).astype(int)] = [np.inf, -np.inf, np.nan, 0, -0.0]
    with np.errstate(all="ignore"):
        expected, = cpu_eval_graph(g.to_bytes(), batch, inputs)
    with CudaExecutor(0, g, batch, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate(inputs)
    if exact:     # (every operation rounds its exact result once, in the kernel and in the oracle)
        np.testing.assert_array_equal(got, expected)
        return
    # an exponential and a quotient, 2 ulp each, behind a sum of two products; of f16 their own roundings and one step more
    finite = np.isfinite(expected)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(expected))
    scale = 4e-3 if expected.dtype == np.float16 else 4e-6
    np.testing.assert_allclose(got[finite].astype(np.float64), expected[finite].astype(np.float64), rtol=scale, atol=max(atol, scale / 4))


@pytest.mark.gpu
@pytest.mark.parametrize("name,dtype,dims,row", CASES)
def test_matches_oracle(name, dtype, dims, row):
    # (the oracle's error function is a polynomial, 3e-7 off, here times x * gate / 2)
    check(program(name, dtype, dims, row), 0, len(dims) + dims[0], name in ("sum", "affine"), atol=4e-6 if name == "geglu" else 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F32, F16])
@pytest.mark.parametrize("rows,heads,d", [(7, 2, 64), (333, 4, 128), (700, 16, 128)])
def test_rotary(rows, heads, d, dtype):
    check(rotary(dtype, rows, heads, d), 2, rows, True)
