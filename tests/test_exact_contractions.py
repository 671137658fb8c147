"""The exact-f32 contraction kernel (KN_MATH_F32) at the edges of its tiles, K blocks and K slices, against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, CudaExecutor
from kyanite_b200.graph import DType, Graph, SliceRange, shape
from oracle.cpu_eval import cpu_eval_graph

pytestmark = pytest.mark.gpu


def check(g, inputs):
    with CudaExecutor(0, g, 0, math_mode=MATH_F32) as ex:
        got = ex.evaluate(inputs)[0].astype(np.float64)
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)[0].astype(np.float64)
    # products and sums are f32 in both, in different orders: n-term sums of O(1) products of size sqrt(n) differ by
    # a few roundings of the running sum, sqrt(n) * sqrt(n) * 2^-24 at most in practice; 1e-5 of the scale covers n <= 8192.
    # f16 results are rounded once more: half an ulp, 2^-11.
    rel = 1e-5 if ex._out_info[0][1] == DType.F32 else 1e-5 + 2.0 ** -11
    assert np.abs(got - expected).max() <= rel * max(1.0, np.abs(expected).max())


# one tile of 64 and its neighbours, K blocks of 32 and their remainders, sliced K, more tiles than two rounds of large ones
@pytest.mark.parametrize("b,m,n,k", [(1, 9, 9, 1), (1, 63, 65, 31), (2, 64, 64, 32), (1, 65, 63, 33), (3, 127, 129, 36), (1, 64, 256, 2048),
                                     (1, 70, 40, 1030), (1, 4700, 1153, 40)])
@pytest.mark.parametrize("layout", ["plain", "transposed", "half"])
def test_matmul(b, m, n, k, layout):
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    dtype = DType.F16 if layout == "half" else DType.F32
    g = Graph()
    if layout == "transposed":   # A along its rows, B along K
        x = g.permute(g.input(shape(b, k, m)), [0, 2, 1])
        w = g.permute(g.input(shape(b, n, k)), [0, 2, 1])
        shapes = [(b, k, m), (b, n, k)]
    else:
        x, w = g.input(shape(b, m, k), dtype), g.input(shape(b, k, n), dtype)
        shapes = [(b, m, k), (b, k, n)]
    g.output(g.batched_mat_mul(x, w))
    check(g, [(rng.standard_normal(s) * (k ** -0.25)).astype(dtype.np) for s in shapes])


# channels that are and are not whole 16-byte chunks or K blocks, strides, taps outside the image, one tile and many
@pytest.mark.parametrize("n,c,hw,k,r,stride,pad", [(1, 128, 8, 128, 3, 1, 1), (3, 21, 9, 70, 3, 1, 1), (2, 33, 7, 5, 5, 2, 2), (1, 4, 3, 3, 1, 1, 0),
                                                   (65, 36, 8, 64, 3, 1, 0), (130, 64, 9, 192, 1, 1, 0)])
@pytest.mark.parametrize("chained", [False, True])
def test_convolution(n, c, hw, k, r, stride, pad, chained):
    rng = np.random.default_rng(n + c + k)
    g = Graph()
    x = g.input(shape(n, c, hw, hw))
    weight = lambda o, i, s: g.constant_tensor((rng.standard_normal((o, i, s, s)) * (i * s * s) ** -0.5).astype(np.float32))  # noqa: E731
    y = g.conv(x, weight(k, c, r), stride, stride, pad, pad)
    y = g.relu(g.add(y, g.constant_tensor(rng.standard_normal((1, k, 1, 1)).astype(np.float32))))
    if chained:   # the first result stays channels-last for the second convolution, and is added to it
        y = g.add(g.conv(y, weight(k, k, 3), 1, 1, 1, 1), y)
    g.output(y)
    check(g, [rng.standard_normal((n, c, hw, hw)).astype(np.float32)])


def sliced(g, base, dims, axis, start):
    """`dims` of `base`, which has `start` + 3 more entries along `axis`, from entry `start` on"""
    return g.slice(base, axis, SliceRange(start, start + dims[axis]))


# One operand in whole 16-byte pieces, the other starting at an odd element: each is fetched in its own way, also where
# nothing is read (rows past the last, taps outside the image, chunks past the end of K).
@pytest.mark.parametrize("dtype", [DType.F32, DType.F16], ids=["f32", "f16"])
@pytest.mark.parametrize("offset", ["a", "b"])
@pytest.mark.parametrize("m,n,k", [(70, 33, 64), (9, 40, 72), (130, 70, 40)])
def test_matmul_with_one_operand_off_16_bytes(m, n, k, offset, dtype):
    rng = np.random.default_rng(m + n + k)
    g = Graph()
    grown = lambda *s: (*s[:-1], s[-1] + 4)  # noqa: E731
    a, b = (1, m, k), (1, n, k)
    shapes = [grown(*a) if offset == "a" else a, grown(*b) if offset == "b" else b]
    x, w = (g.input(shape(*s), dtype) for s in shapes)
    if offset == "a":
        x = sliced(g, x, a, 2, 1)
    else:
        w = sliced(g, w, b, 2, 1)
    g.output(g.batched_mat_mul(x, g.permute(w, [0, 2, 1])))
    check(g, [(rng.standard_normal(s) * k ** -0.25).astype(dtype.np) for s in shapes])


def test_matmul_of_a_column_slice():
    """x[70, 64] . w[:, 1:33]: B along its rows, its first element 4 bytes past an aligned address"""
    rng = np.random.default_rng(5)
    g = Graph()
    x, w = g.input(shape(1, 70, 64)), g.input(shape(1, 64, 41))
    g.output(g.batched_mat_mul(x, sliced(g, w, (1, 64, 32), 2, 1)))
    check(g, [rng.standard_normal((1, 70, 64)).astype(np.float32), rng.standard_normal((1, 64, 41)).astype(np.float32)])


@pytest.mark.parametrize("offset", ["image", "filter", "flipped"])
def test_convolution_with_one_operand_off_16_bytes(offset):
    rng = np.random.default_rng(6)
    g = Graph()
    image, weight = (1, 8, 9, 9), (20, 8, 3, 3)
    x = g.input(shape(1, 8, 9, 13) if offset == "image" else shape(*image))
    w = g.input(shape(20, 12, 3, 3) if offset != "image" else shape(*weight))
    inputs = [rng.standard_normal([d.eval(0) for d in g[v].shape]).astype(np.float32) for v in (x, w)]
    if offset == "image":
        x = sliced(g, x, image, 3, 1)
    else:
        w = sliced(g, w, weight, 1, 1)
        x = g.flip(x, 2) if offset == "flipped" else x
    g.output(g.conv(x, w, 1, 1, 1, 1))
    check(g, inputs)


# nothing to sum: zeros, and what the epilogue adds to them
@pytest.mark.parametrize("dtype", [DType.F32, DType.F16], ids=["f32", "f16"])
def test_empty_matmul(dtype):
    g = Graph()
    y = g.batched_mat_mul(g.input(shape(2, 70, 0), dtype), g.input(shape(2, 0, 9), dtype))
    bias = np.arange(9).astype(dtype.np).reshape(1, 1, 9)
    g.output_all([y, g.add(y, g.constant_tensor(bias))])
    with CudaExecutor(0, g, 0, math_mode=MATH_F32) as ex:
        zeros, biased = ex.evaluate([np.zeros((2, 70, 0), dtype.np), np.zeros((2, 0, 9), dtype.np)])
    np.testing.assert_array_equal(zeros, np.zeros((2, 70, 9)))
    np.testing.assert_array_equal(biased, np.broadcast_to(bias, (2, 70, 9)))


def test_empty_convolution():
    g = Graph()
    y = g.conv(g.input(shape(2, 0, 5, 5)), g.input(shape(70, 0, 3, 3)), 1, 1, 1, 1)
    bias = np.arange(70).astype(np.float32).reshape(1, 70, 1, 1)
    g.output(g.add(y, g.constant_tensor(bias)))
    with CudaExecutor(0, g, 0, math_mode=MATH_F32) as ex:
        got, = ex.evaluate([np.zeros((2, 0, 5, 5), np.float32), np.zeros((70, 0, 3, 3), np.float32)])
    np.testing.assert_array_equal(got, np.broadcast_to(bias, (2, 70, 5, 5)))


@pytest.mark.parametrize("dtype,k,side", [(DType.F32, 1 << 29, 9), (DType.F16, 1 << 30, 1)], ids=["f32", "f16"])
def test_long_reduction(dtype, k, side):
    """Rows of 2 GB: byte counts along K do not fit 32 bits.  One entry in 2^20 is not zero, so every sum is exact."""
    period = 1 << 20
    pattern = np.zeros((1, period), dtype.np)
    pattern[0, 12345] = 1
    g = Graph()
    row = g.add(g.broadcast(g.constant_tensor(pattern), shape(k // period, period)), g.broadcast(g.view(g.input(shape(1), dtype), shape(1, 1)), shape(k // period, period)))
    row = g.broadcast(g.view(row, shape(1, 1, k)), shape(1, side, k))
    g.output(g.batched_mat_mul(row, g.permute(row, [0, 2, 1])))
    with CudaExecutor(0, g, 0, math_mode=MATH_F32) as ex:
        got, = ex.evaluate([np.zeros(1, dtype.np)])
    np.testing.assert_array_equal(got, np.full((1, side, side), k // period))


# B along its columns: tiles of 32 and of 64, with and without slices of K (3, 7 and 8 of them), K blocks that end inside a
# slice, rows of A and of B that are and are not whole 16-byte pieces, columns past the last tile
@pytest.mark.parametrize("b,m,n,k", [(1, 64, 128, 1152), (1, 33, 36, 930), (12, 120, 64, 120), (2, 1024, 80, 77), (1, 4096, 128, 420), (1, 2050, 190, 1040),
                                     (1, 31, 30, 33), (30, 63, 65, 64)])
@pytest.mark.parametrize("addend", [False, True])
def test_matmul_along_columns(b, m, n, k, addend):
    rng = np.random.default_rng(m + n + k)
    g = Graph()
    y = g.batched_mat_mul(g.input(shape(b, m, k)), g.input(shape(b, k, n)))
    if addend:
        y = g.relu(g.add(g.add(y, g.constant_tensor(rng.standard_normal((1, 1, n)).astype(np.float32))), g.input(shape(b, m, n))))
    g.output(y)
    shapes = [(b, m, k), (b, k, n)] + ([(b, m, n)] if addend else [])
    check(g, [(rng.standard_normal(s) * (k ** -0.25 if i < 2 else 1)).astype(np.float32) for i, s in enumerate(shapes)])


# a filter laid out along its output channels at planning time, results along channels and along positions
@pytest.mark.parametrize("n,c,k,hw", [(1, 128, 128, 8), (1, 21, 70, 9), (64, 40, 128, 8), (2, 64, 34, 7)])
def test_convolution_chain_of_few_positions(n, c, k, hw):
    rng = np.random.default_rng(n + c + k)
    g = Graph()
    weight = lambda o, i, s: g.constant_tensor((rng.standard_normal((o, i, s, s)) * (i * s * s) ** -0.5).astype(np.float32))  # noqa: E731
    y = g.relu(g.conv(g.input(shape(n, c, hw, hw)), weight(k, c, 3), 1, 1, 1, 1))
    y = g.relu(g.add(g.conv(y, weight(k, k, 3), 1, 1, 1, 1), y))
    g.output(g.conv(y, weight(5, k, 1), 1, 1, 0, 0))
    check(g, [rng.standard_normal((n, c, hw, hw)).astype(np.float32)])
