"""Runs of 3x3 convolutions in exact f32 as one launch (kernels/conv_chain_exact.cu), at every number of CTAs per image."""
import numpy as np
import pytest

from kyanite_b200.executor import FLAG_NO_CONV_CHAIN, MATH_F32, MATH_TF32, plan_describe
from oracle.cpu_eval import cpu_eval_graph
from kyanite_b200.graph import BATCH, Graph, shape
from test_conv_chain import rng, steps, tower


def chains(g, batch, mode=MATH_F32, flags=0):
    return [l for l in steps(plan_describe(g, batch, mode, flags=flags)) if "ConvChain" in l]


@pytest.mark.parametrize("channels,batch,ctas", [(128, 7, 16), (128, 12, 8), (128, 33, 4), (128, 45, 2), (128, 74, 2), (128, 148, 1), (64, 1, 8), (64, 16, 4), (32, 34, 2)])
def test_ctas_per_image(channels, batch, ctas):
    g = tower(channels, 2, 8, 8, 21)
    line, = chains(g, batch)
    assert f"exact, {ctas} CTAs per image" in line and "/tc" not in line
    assert not chains(g, batch, flags=FLAG_NO_CONV_CHAIN)


def test_route():
    assert not chains(tower(128, 2, 8, 8, 21), 149)                          # more images than one round
    for batch in (11, 40, 110):                                              # wide layers, a round of which little is used
        assert not chains(tower(128, 2, 8, 8, 21), batch)
    assert not chains(tower(128, 2, 16, 8, 21), 5) and chains(tower(128, 2, 16, 8, 21), 6)
    assert not chains(tower(128, 2, 7, 7, 21), 130) and chains(tower(128, 2, 7, 7, 21), 146)
    assert not chains(tower(64, 1, 8, 8, 21), 4)                             # three layers
    assert chains(tower(64, 2, 8, 8, 21), 1, MATH_TF32)                      # fewer than 128 positions keep f32 operands
    assert not chains(tower(36, 2, 8, 8, 21), 4)                             # channels that are no multiple of eight
    assert not chains(tower(64, 2, 9, 9, 21), 4)                             # rows that are too long


CASES = [  # channels, input channels, blocks, h, w, batch
    (128, 21, 2, 8, 8, 6), (128, 128, 2, 8, 8, 7), (128, 5, 2, 8, 8, 12), (128, 21, 2, 8, 8, 25), (128, 21, 2, 8, 8, 50), (128, 3, 2, 8, 8, 120),
    (64, 21, 2, 7, 7, 2), (64, 64, 2, 8, 8, 12), (64, 9, 2, 16, 8, 3), (64, 1, 2, 8, 8, 75), (96, 30, 2, 7, 7, 33), (32, 100, 2, 8, 7, 20), (40, 1, 2, 5, 8, 90),
]


@pytest.mark.gpu
@pytest.mark.parametrize("channels,c_in,blocks,h,w,batch", CASES)
@pytest.mark.parametrize("residual", [True, False])
def test_matches_oracle(channels, c_in, blocks, h, w, batch, residual):
    from kyanite_b200.executor import CudaExecutor
    g = tower(channels, blocks, h, w, c_in, seed=channels + h, residual=residual, relu=residual)
    assert chains(g, batch)
    x = rng(c_in).standard_normal((batch, c_in, h, w)).astype(np.float32)
    expected, = cpu_eval_graph(g.to_bytes(), batch, [x])
    with CudaExecutor(0, g, batch, math_mode=MATH_F32) as ex:
        got, = ex.evaluate([x])
        # five layers of f32 sums of up to 1152 terms in another order: 1e-5 of the scale
        assert np.abs(got.astype(np.float64) - expected).max() <= 1e-5 * np.abs(expected).max()
        np.testing.assert_array_equal(got, ex.evaluate([x])[0])


@pytest.mark.gpu
@pytest.mark.parametrize("channels,c_in,batch", [(48, 60, 100), (40, 64, 90), (80, 100, 70), (96, 128, 30), (128, 21, 7)])
def test_infinity_reaches_its_neighbours_only(channels, c_in, batch):
    """Positive weights and no activation: within reach of an infinity every channel is infinite, nothing is NaN.  (Whole chunks of
    weights go past the channels of the trunk in most of these.)"""
    from kyanite_b200.executor import CudaExecutor
    g, layers = Graph(), 4
    cur = g.input(shape(BATCH, c_in, 8, 8))
    for c in [c_in] + [channels] * (layers - 1):
        cur = g.conv(cur, g.constant_tensor(np.full((channels, c, 3, 3), 0.125, np.float32)), 1, 1, 1, 1)
    g.output(cur)
    assert chains(g, batch)
    x = np.ones((batch, c_in, 8, 8), np.float32)
    x[3, min(channels, c_in - 1), 1, 7] = np.inf      # (the first channel behind the trunk's)
    want = np.zeros((batch, channels, 8, 8), bool)
    want[3, :, :6, 3:] = True
    with CudaExecutor(0, g, batch, math_mode=MATH_F32) as ex:
        got, = ex.evaluate([x])
    np.testing.assert_array_equal(got == np.inf, want)
    assert np.isfinite(got[~want]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("channels,batch", [(128, 130), (128, 46), (128, 25), (128, 12), (128, 7), (64, 46)])
def test_no_further_from_64_bits_than_one_by_one(channels, batch):
    """Five layers; as many sums are compared as make the ratio repeat to 2 % from one set of weights to the next."""
    from kyanite_b200.executor import CudaExecutor
    g = tower(channels, 2, 8, 8, 21, seed=channels + batch)
    assert chains(g, batch)
    x = rng(batch).standard_normal((batch, 21, 8, 8)).astype(np.float32)
    results = []
    for flags in (0, FLAG_NO_CONV_CHAIN):
        with CudaExecutor(0, g, batch, math_mode=MATH_F32, flags=flags) as ex:
            results.append(ex.evaluate([x])[0].astype(np.float64))
    want = in_64_bits(g, x)
    chain, single = (np.sqrt(((r - want) ** 2).mean()) for r in results)
    assert chain <= 1.03 * single


def in_64_bits(g, x):
    """The graph of `tower`: convolutions, sums and ReLUs, node by node."""
    from kyanite_b200.graph import BinaryOp, OpKind
    values = g.all_values()
    at = {}
    for i, v in enumerate(values):
        info = g[v]
        a = [at[k] for k in info.inputs]
        if info.kind == OpKind.INPUT:
            y = x.astype(np.float64)
        elif info.kind == OpKind.CONSTANT:
            y = np.asarray(info.tensor, np.float64)
        elif info.kind == OpKind.CONV:
            padded = np.pad(a[0], ((0, 0), (0, 0), (1, 1), (1, 1)))
            windows = np.lib.stride_tricks.sliding_window_view(padded, (3, 3), (2, 3))
            y = np.einsum("nchwrs,kcrs->nkhw", windows, a[1], optimize=True)
        elif info.kind in (OpKind.BROADCAST, OpKind.VIEW):
            y = a[0] if a[0].ndim == 4 else a[0].reshape([1] * 4)
        else:
            y = {BinaryOp.ADD: np.add, BinaryOp.MAX: np.maximum, BinaryOp.MIN: np.minimum}[info.binary_op](a[0], a[1])
        at[i] = y
    return at[values.index(g.outputs[0])]
