"""Convolutions of a long reduction to fewer than 16 channels, at few positions: slices of K over clusters (kernels/gemm_persistent.cu),
which of them the planner routes there, and their values against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_F32, MATH_TF32, CudaExecutor, plan_describe
from kyanite_b200.graph import BATCH, Graph, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph


def graph(c, k, h, w, skip=False):
    rng = np.random.default_rng(c + k + h)
    g = Graph()
    y = g.conv(g.input(shape(BATCH, c, h, w)), g.constant_tensor((rng.standard_normal((k, c, 3, 3)) / np.sqrt(9 * c)).astype(np.float32)), 1, 1, 1, 1)
    y = g.add(y, g.constant_tensor(rng.standard_normal((1, k, 1, 1)).astype(np.float32)))
    g.output(g.relu(g.add(y, g.input(shape(BATCH, k, h, w)))) if skip else y)
    return g


def sliced(c, k, h, w, batch=1, mode=MATH_TF32):
    return "matmul b=%d m=%d " % (batch, k) in plan_describe(graph(c, k, h, w), batch, mode)


def test_route():
    assert sliced(256, 4, 64, 64) and sliced(256, 12, 16, 32, 2) and sliced(256, 8, 74, 128)
    assert not sliced(256, 4, 75, 128)          # the convolution kernel has CTAs for half of the SMs
    assert not sliced(256, 4, 64, 64, 3)
    assert not sliced(256, 6, 64, 64)           # channels that are no whole 16-byte pieces of the filter's rows
    assert not sliced(64, 4, 64, 64)            # a short reduction
    assert not sliced(256, 4, 12, 16)           # positions that are no whole tiles
    assert not sliced(256, 4, 64, 64, 1, MATH_F32)


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(256, 4, 64, 64, 1, False), (320, 4, 64, 64, 1, True), (256, 12, 16, 32, 2, True), (256, 8, 74, 128, 1, False), (512, 4, 8, 16, 3, False),
                                  (256, 4, 2, 64, 1, True)])
def test_values(case):
    g = graph(*case[:4], case[5])
    batch = case[4]
    rng = np.random.default_rng(1)
    inputs = [rng.standard_normal([d.eval(batch) for d in g[v].shape]).astype(np.float32) for v in g.inputs]
    expected = cpu_eval_graph(g.to_bytes(), batch, inputs)
    with CudaExecutor(0, g, batch, math_mode=MATH_TF32) as ex:
        # TF32 operands, sums of up to 4608 products (as the other convolutions of this route)
        assert_tensors_match(expected, ex.evaluate(inputs), 4e-3, 4e-3, abs_scaled=True)
