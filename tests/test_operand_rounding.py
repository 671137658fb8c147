"""Which calls of the default mode (KN_MATH_TF32) round f32 operands to TF32's 11 bits, and which keep them: convolutions over
less than a tile of positions, attention and joined projections whose matmuls by themselves would keep them.  The reference computes its matmuls in f32 throughout
(kn-cuda-sys/src/wrapper/group.rs:120-171)."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import Graph, shape
from oracle.cpu_eval import cpu_eval_graph


def rng(seed, *s):
    return np.random.Generator(np.random.PCG64(seed)).standard_normal(s).astype(np.float32)


def contractions(g):
    """(on the tensor cores, on the exact kernel)"""
    kinds = [line.split()[2] for line in plan_describe(g, 0, MATH_TF32).splitlines() if line.startswith("step")]
    kinds = [k for k in kinds if k.startswith(("Conv", "Gemm"))]
    return sum(not k in ("Conv", "Gemm") for k in kinds), sum(k in ("Conv", "Gemm") for k in kinds)


def check_exact(g):
    from kyanite_b200.executor import CudaExecutor
    inputs = [rng(7 + i, *[d.eval(0) for d in g[v].shape]) for i, v in enumerate(g.inputs)]
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)
    for e, o in zip(cpu_eval_graph(g.to_bytes(), 0, inputs), got):
        # f32 products and sums in another order: 1e-5 of the scale for reductions of up to 8192 terms, a thirtieth of what
        # rounding the operands to 11 bits moves them by
        assert np.abs(o.astype(np.float64) - e).max() <= 1e-5 * np.abs(e).max()


def tower(images, side, channels, layers=3):
    g = Graph()
    y = g.input(shape(images, channels, side, side))
    for i in range(layers):
        w = g.constant_tensor(rng(i, channels, channels, 3, 3) / np.float32(3 * channels ** 0.5))
        y = g.relu(g.add(g.conv(y, w, 1, 1, 1, 1), g.constant_tensor(rng(10 + i, 1, channels, 1, 1))))
    g.output(y)
    return g


# positions: 64, 81, 127; 128 and more go to the tensor cores as ever
SMALL = [(1, 8, 128), (1, 9, 64), (127, 1, 64), (2, 7, 33)]


def test_convolution_route():
    for case in SMALL:
        assert contractions(tower(*case)) == (0, 3), case
    assert contractions(tower(2, 8, 128))[1] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("case", SMALL)
def test_small_convolutions_keep_f32(case):
    check_exact(tower(*case))


def attention(b, m, n, k, dv, masked=False, along_keys=False):
    g = Graph()
    q, keys = g.input(shape(b, m, k)), g.input(shape(b, n, k))
    v = g.permute(g.input(shape(b, dv, n)), [0, 2, 1]) if along_keys else g.input(shape(b, n, dv))
    scores = g.mul(g.batched_mat_mul(q, g.permute(keys, [0, 2, 1])), g.scalar(0.3))
    if masked:
        scores = g.add(scores, g.constant_tensor(np.triu(np.full((1, m, n), -np.inf, np.float32), 1)))
    g.output(g.batched_mat_mul(g.softmax(scores, 2), v))
    return g


# fewer rows than the tensor-core matmul takes, masked and not, ragged and whole 16-byte rows
FEW_ROWS = [(3, 63, 77, 40, 40), (2, 20, 300, 64, 64), (1, 16, 16, 8, 8), (12, 48, 48, 64, 64)]


def test_attention_route():
    for case in FEW_ROWS:
        for masked in (False, True):
            assert contractions(attention(*case, masked)) == (0, 2), case
    # 64 rows and more: the scores on the tensor cores, the small second matmul with f32 probabilities and values as ever
    assert contractions(attention(12, 120, 120, 64, 64)) == (1, 1)
    assert contractions(attention(12, 120, 120, 64, 64, along_keys=True)) == (1, 0)
    assert contractions(attention(120, 120, 120, 64, 64)) == (1, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("case", FEW_ROWS)
def test_attention_of_few_rows_keeps_f32(case, masked):
    check_exact(attention(*case, masked))


def projections(m, k, widths, n_major):
    """x . W_i for constant W_i [k, n_i] (n_major: [n_i, k], transposed), each read by a small matmul of its own"""
    g = Graph()
    x = g.input(shape(1, m, k))
    for i, n in enumerate(widths):
        if n_major:
            w = g.permute(g.constant_tensor(rng(i, 1, n, k)), [0, 2, 1])
        else:
            w = g.constant_tensor(rng(i, 1, k, n))
        y = g.batched_mat_mul(x, w)
        g.output(g.batched_mat_mul(g.permute(y, [0, 2, 1]), g.input(shape(1, m, 4))))
    return g


# weights along their columns and too little work for a copy; a width below what the tensor cores take; few rows
SEPARATE = [(87, 336, [84, 96], False), (122, 104, [36, 28, 4], True), (40, 64, [64, 64], True)]


def test_projection_route():
    for case in SEPARATE[:2]:
        assert "projections of one tensor" not in plan_describe(projections(*case), 0, MATH_TF32), case
    assert "2 projections of one tensor" in plan_describe(projections(120, 768, [768, 768], True), 0, MATH_TF32)


@pytest.mark.gpu
@pytest.mark.parametrize("case", [SEPARATE[0], SEPARATE[2]])
def test_small_projections_keep_f32(case):
    check_exact(projections(*case))
