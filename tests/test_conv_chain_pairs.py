"""The convolution chain on CTA pairs (kernels/conv_chain_pair.cu): which images it takes, and its results at the sizes where its
layout changes.  Bounds: those of test_conv_chain.py (operands rounded to TF32, sums in f32)."""
import numpy as np
import pytest

from kyanite_b200.configs import resnet_tower
from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, Graph, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph
from test_conv_chain import rng, steps, tower, tower_with_heads


@pytest.mark.parametrize("h,w,pairs", [(8, 8, True), (9, 9, True), (11, 10, True), (11, 11, False), (12, 12, False), (16, 8, True), (17, 8, False)])
def test_which_images_run_on_pairs(h, w, pairs):
    chains = [l for l in steps(plan_describe(tower(32, 1, h, w, 8), 8, MATH_TF32)) if "ConvChain" in l]
    assert chains and all(("on CTA pairs" in l) == pairs for l in chains)


CASES = [  # channels, input channels, h, w, batch, heads
    (128, 21, 8, 8, 3, [73, 32]),      # two boards a CTA in rows of eight, one of the pair's four missing
    (128, 128, 8, 8, 7, [5]),          # the chain's input is added
    (128, 16, 16, 8, 3, [128]),        # one image of sixteen groups
    (64, 8, 5, 8, 23, [100]),          # three images side by side, fifteen groups
    (64, 100, 7, 7, 9, [9, 3]),        # an input wider than the trunk
    (48, 5, 9, 9, 5, [17]),            # half a channel block
    (16, 2, 5, 6, 33, [40, 7]),        # one block, a pointwise layer wider than the trunk
    (96, 3, 11, 10, 2, []),            # 120 of 128 lanes
    (20, 4, 4, 4, 70, []),             # several rows of images
    (128, 4, 12, 12, 3, [6]),          # the other kernel: one image per CTA
    (32, 30, 12, 11, 5, []),
]


@pytest.mark.gpu
@pytest.mark.parametrize("channels,c_in,h,w,batch,heads", CASES)
@pytest.mark.parametrize("trunk", [False, True])
def test_pairs_match_oracle(channels, c_in, h, w, batch, heads, trunk):
    from kyanite_b200.executor import CudaExecutor
    if heads:
        g = tower_with_heads(channels, h, w, c_in, heads, [i % 2 == 0 for i in range(len(heads))], trunk_output=trunk, seed=h + w)
    else:
        g = tower(channels, 2, h, w, c_in, seed=h + w, residual=trunk, relu=trunk)
    assert any("ConvChain" in l for l in steps(plan_describe(g, batch, MATH_TF32)))
    x = rng(c_in).standard_normal((batch, c_in, h, w)).astype(np.float32)
    expected = cpu_eval_graph(g.to_bytes(), batch, [x])
    with CudaExecutor(0, g, batch, math_mode=MATH_TF32) as ex:
        got = ex.evaluate([x])
        assert_tensors_match(expected, got, 4e-3, 4e-3, abs_scaled=True)
        for a, b in zip(got, ex.evaluate([x])):
            np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
def test_infinity_and_nan_stay_in_their_image():
    from kyanite_b200.executor import CudaExecutor
    r, g = rng(2), Graph()
    cur = g.input(shape(BATCH, 8, 8, 8))
    for c in (8, 64):   # (without an activation: a ReLU makes zero of NaN)
        cur = g.conv(cur, g.constant_tensor((r.standard_normal((64, c, 3, 3)) / 20).astype(np.float32)), 1, 1, 1, 1)
    g.output(cur)
    assert any("on CTA pairs" in l for l in steps(plan_describe(g, 9, MATH_TF32)))
    x = rng(1).standard_normal((9, 8, 8, 8)).astype(np.float32)
    with CudaExecutor(0, g, 9, math_mode=MATH_TF32) as ex:
        clean, = ex.evaluate([x])
        x[4, 2, 3, 3] = np.nan
        x[7, 1, 0, 7] = np.inf
        got, = ex.evaluate([x])
    others = [i for i in range(9) if i not in (4, 7)]
    np.testing.assert_array_equal(got[others], clean[others])
    assert not np.isfinite(got[4][:, 2:5, 2:5]).any() and not np.isfinite(got[7][:, 0:2, 6:8]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("channels,c_in", [(48, 60), (20, 8), (40, 64), (64, 100), (128, 128), (12, 3)])
def test_infinity_reaches_its_neighbours_only(channels, c_in):
    """Positive weights and no activation: within reach of an infinity every channel is infinite, nothing is NaN."""
    from kyanite_b200.executor import CudaExecutor
    g, layers = Graph(), 3
    cur = g.input(shape(BATCH, c_in, 8, 8))
    for c in [c_in] + [channels] * (layers - 1):
        cur = g.conv(cur, g.constant_tensor(np.full((channels, c, 3, 3), 0.125, np.float32)), 1, 1, 1, 1)
    g.output(cur)
    assert any("on CTA pairs" in l for l in steps(plan_describe(g, 5, MATH_TF32)))
    x = np.ones((5, c_in, 8, 8), np.float32)
    x[3, c_in - 1, 2, 7] = np.inf
    want = np.zeros((5, channels, 8, 8), bool)
    want[3, :, :6, 4:] = True
    with CudaExecutor(0, g, 5, math_mode=MATH_TF32) as ex:
        got, = ex.evaluate([x])
    np.testing.assert_array_equal(got == np.inf, want)
    assert np.isfinite(got[~want]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("channels", [16, 32, 72, 128])
def test_every_layer_adds_its_own_bias(channels):
    """Identity filters and small whole biases: each layer's bias counts, exactly, also with two executors at work at a time (the
    table of biases in shared memory is written while earlier rows of it are read)."""
    from kyanite_b200.executor import CudaExecutor
    r, g, layers = rng(channels), Graph(), 30
    biases = r.integers(-9, 10, (layers, channels)).astype(np.float32)
    w = np.zeros((channels, channels, 3, 3), np.float32)
    w[range(channels), range(channels), 1, 1] = 1
    cur = g.input(shape(BATCH, channels, 8, 8))
    for b in biases:
        cur = g.add(g.conv(cur, g.constant_tensor(w), 1, 1, 1, 1), g.constant_tensor(b.reshape(1, channels, 1, 1)))
    g.output(cur)
    assert any("on CTA pairs" in l and "layers=%d" % layers in l for l in steps(plan_describe(g, 300, MATH_TF32)))
    x = r.integers(-9, 10, (300, channels, 8, 8)).astype(np.float32)
    want = x + biases.sum(0).reshape(1, channels, 1, 1)    # (at most 280: exact in TF32)
    with CudaExecutor(0, g, 300, math_mode=MATH_TF32) as a, CudaExecutor(0, g, 300, math_mode=MATH_TF32) as b:
        for _ in range(20):
            a.evaluate_begin([x])
            b.evaluate_begin([x])
            np.testing.assert_array_equal(a.evaluate_end()[0], want)
            np.testing.assert_array_equal(b.evaluate_end()[0], want)


def test_heads_of_large_batches_join_the_chain():
    """A 1x1 convolution large enough to be a matmul of its own stays with the chain whose result it reads, if all of them fit."""
    g, _ = resnet_tower()
    d = steps(plan_describe(g, 2048, MATH_TF32))
    assert "heads=73+32 (trunk result not stored)" in d[0] and len(d) == 5
    d = steps(plan_describe(tower_with_heads(128, 8, 8, 8, [100, 40], [False] * 2), 2048, MATH_TF32))
    assert len([l for l in d if "conv via im2col" in l]) == 2 and "heads=" not in d[0]
