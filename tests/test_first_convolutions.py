"""Convolutions of up to eight channels at many positions, as windows (im2col, written a position and tap per thread) and a matmul: which
of them, and their values against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, MATH_TF32, CudaExecutor, plan_describe
from kyanite_b200.graph import BATCH, Graph, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph


def graph(c, k, h, w, r=3, s=3, pad=(1, 1), turned=False, relu=False):
    rng = np.random.default_rng(c + k + h)
    g = Graph()
    x = g.input(shape(BATCH, h, w, c) if turned else shape(BATCH, c, h, w))
    if turned:   # the caller's image has its channels last
        x = g.permute(x, [0, 3, 1, 2])
    y = g.conv(x, g.constant_tensor((rng.standard_normal((k, c, r, s)) / np.sqrt(r * s * c)).astype(np.float32)), 1, 1, *pad)
    y = g.add(y, g.constant_tensor(rng.standard_normal((1, k, 1, 1)).astype(np.float32)))
    g.output(g.relu(y) if relu else y)
    return g


def windows(*args, batch=1, mode=MATH_TF32):
    return " Im2col " in plan_describe(graph(*args), batch, mode)


def test_route():
    assert windows(4, 320, 64, 64) and windows(3, 64, 32, 32) and windows(1, 32, 28, 28) and windows(8, 16, 28, 28, 5, 5, (2, 2))
    assert not windows(9, 64, 32, 32)           # more channels: the convolution kernel reads them from the image
    assert not windows(4, 64, 27, 29)           # fewer positions, as on boards
    assert not windows(8, 64, 32, 32, 7, 7, (3, 3))     # windows of more than 256 elements
    assert not windows(4, 12, 64, 64) and not windows(4, 30, 64, 64)
    assert not windows(4, 64, 64, 64, mode=MATH_F32)
    assert windows(3, 64, 224, 224, batch=16) and windows(8, 64, 64, 64, 7, 7, (3, 3), batch=8)   # 87 and 51 MB of windows
    assert not windows(4, 64, 512, 512, batch=8)        # 302 MB: the limit is 256


CASES = [(4, 320, 64, 64, 3, 3, (1, 1), False, False, 1), (3, 64, 32, 32, 3, 3, (1, 1), False, True, 3), (1, 32, 28, 28, 5, 5, (2, 2), False, False, 2),
         (8, 16, 33, 40, 3, 5, (0, 3), False, True, 2), (5, 20, 31, 29, 7, 1, (3, 0), False, False, 1), (3, 64, 40, 32, 3, 3, (1, 1), True, True, 2),
         (2, 100, 30, 30, 1, 3, (0, 1), False, False, 1), (6, 48, 1, 800, 1, 9, (0, 4), False, False, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_values(case):
    g = graph(*case[:-1])
    batch = case[-1]
    inputs = [np.random.default_rng(1).standard_normal([d.eval(batch) for d in g[v].shape]).astype(np.float32) for v in g.inputs]
    expected = cpu_eval_graph(g.to_bytes(), batch, inputs)
    with CudaExecutor(0, g, batch, math_mode=MATH_TF32) as ex:
        # TF32 operands (2^-11 each), windows of at most 256 products of about unit variance together
        assert_tensors_match(expected, ex.evaluate(inputs), 4e-3, 4e-3, abs_scaled=True)
