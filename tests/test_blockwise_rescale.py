"""Attention by key blocks where every block raises the rows' maxima, so that the output accumulated so far is rescaled while the
block before may still be added to it; numbers of keys at the edges of a block of 64, one and two buffers for keys and values."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import DType, Graph, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph


@pytest.mark.gpu
# (a wide head in f32 over whole blocks of keys goes another way)
# (f32 goes this way where its matmuls by themselves would round their operands; 20 entries leave an SM one CTA, whose softmax warps
# take two blocks at a time)
@pytest.mark.parametrize("n,b,half,d,dv", [(n, *c) for n in (63, 64, 65, 128, 129, 191, 449)
                                           for c in ((220, False, 40, 40), (220, False, 128, 96), (20, True, 128, 128), (20, True, 24, 72), (100, True, 128, 128), (100, True, 24, 72))
                                           if n % 64 or c != (220, False, 128, 96)])
def test_rising_maxima(n, b, half, d, dv):
    from kyanite_b200.executor import CudaExecutor
    m = 200
    dtype = DType.F16 if half else DType.F32
    r = np.random.Generator(np.random.PCG64(n))
    g = Graph()
    q, keys, v = (g.input(shape(*s), dtype) for s in ((b, m, d), (b, n, d), (b, n, dv)))
    g.output(g.batched_mat_mul(g.softmax(g.mul(g.batched_mat_mul(q, g.permute(keys, [0, 2, 1])), g.scalar(1.0, dtype)), 2), v))
    assert any("blockwise-attention" in l for l in plan_describe(g, 0, MATH_TF32).splitlines())
    # scores rise by 12 from block to block (the reference moves by 8 and more in powers of two), falling for every third row
    rising = np.arange(n) // 64 * 12.0
    inputs = [0.2 * r.standard_normal((b, m, d)), 0.2 * r.standard_normal((b, n, d)), r.standard_normal((b, n, dv))]
    inputs[0][:, :, 0] = np.where(np.arange(m) % 3 == 0, -1, 1)
    inputs[1][:, :, 0] = rising
    inputs = [x.astype(dtype.np) for x in inputs]
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)
    # operands of 11 bits: a score of up to 84 is off by 2^-6 in f16 (the oracle rounds it) and its exponential by that much
    assert_tensors_match(expected, got, 2e-2 if half else 4e-3, 2e-2 if half else 4e-3, abs_scaled=True)


@pytest.mark.gpu
@pytest.mark.parametrize("half", [False, True])
def test_scores_of_minus_infinity_behind_masked_keys(half):
    """A mask of the type's lowest value over the first keys of some rows, then keys that are not masked at all but whose scores are
    -infinity for them: those rows are the mean of the masked keys' values."""
    from kyanite_b200.executor import CudaExecutor
    b, m, n, d = (20, 256, 256, 64) if half else (220, 256, 256, 40)
    dtype = DType.F16 if half else DType.F32
    r = np.random.Generator(np.random.PCG64(3))
    g = Graph()
    q, keys, v = (g.input(shape(*s), dtype) for s in ((b, m, d), (b, n, d), (b, n, d)))
    mask = np.zeros((1, m, n), dtype.np)
    mask[:, 64:200:3, :128] = np.finfo(dtype.np).min
    scores = g.mul(g.batched_mat_mul(q, g.permute(keys, [0, 2, 1])), g.scalar(0.25, dtype))
    g.output(g.batched_mat_mul(g.softmax(g.add(scores, g.broadcast(g.constant_tensor(mask), shape(b, m, n))), 2), v))
    assert any("blockwise-attention" in l for l in plan_describe(g, 0, MATH_TF32).splitlines())
    inputs = [0.3 * r.standard_normal((b, m, d)), 0.3 * r.standard_normal((b, n, d)), r.standard_normal((b, n, d))]
    inputs[0][:, :, 0] = 1
    inputs[1][:, 128:, 0] = -np.inf
    inputs = [x.astype(dtype.np) for x in inputs]
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate(inputs)
    want = np.broadcast_to(inputs[2][:, None, :128].astype(np.float64).mean(2), (b, m, d))
    rows = range(64, 200, 3)
    # (the mean of 128 values with operands of 11 bits; masked scores are the lowest value whatever the score)
    assert np.abs(got[:, rows].astype(np.float64) - want[:, rows]).max() <= 4e-3
    assert np.isfinite(got).all()
