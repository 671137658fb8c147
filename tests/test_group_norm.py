"""Group normalisation with scale, shift and SiLU as one step (kernels/group_norm.cu): what is matched, and its values for plain and
channels-last tensors, groups of any number of channels, on one to eight CTAs."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, Graph, UnaryOp, shape


def rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def norm(g, t, c, groups, h, w, silu, seed=0, swapped=False):
    r = rng(seed)
    gamma, beta = (g.constant_tensor((a + 0.3 * r.standard_normal((1, c, 1, 1))).astype(np.float32)) for a in (1, 0))
    n = g.view(g.layernorm(g.view(t, shape(BATCH, groups, c // groups * h * w)), 2, 1e-5), shape(BATCH, c, h, w))
    y = g.add(beta, g.mul(gamma, n)) if swapped else g.add(g.mul(n, gamma), beta)
    return g.mul(y, g.unary(UnaryOp.SIGMOID, y)) if silu else y


def conv(g, t, cin, cout, seed):
    w = (rng(seed).standard_normal((cout, cin, 3, 3)) / np.sqrt(9 * cin)).astype(np.float32)
    return g.conv(t, g.constant_tensor(w), 1, 1, 1, 1)


def build(c, groups, h, w, silu, before, after):
    """[3x3 convolution ->] group norm [-> 3x3 convolution]; outputs: what the norm reads, the norm, the convolution behind it"""
    g = Graph()
    x = g.input(shape(BATCH, c, h, w))
    if before:
        x = conv(g, x, c, c, 1)
    y = norm(g, x, c, groups, h, w, silu, swapped=silu)
    if before:
        g.output(x)
    g.output(y)
    if after:
        g.output(conv(g, y, c, c, 2))
    return g


def lines(g, batch):
    return [l for l in plan_describe(g, batch, MATH_TF32).splitlines() if l.startswith("step") and " GroupNorm " in l]


CASES = [  # n, c, groups, h, w, silu, convolution before, after
    (2, 40, 4, 16, 12, True, False, False),      # plain to plain
    (1, 12, 4, 66, 64, False, False, False),     # a last CTA with less to do
    (40, 16, 4, 8, 8, True, False, True),        # one CTA a group
    (3, 40, 4, 20, 18, True, False, True),       # plain to channels-last, tiles that are not full
    (1, 96, 3, 16, 16, False, False, True),
    (2, 320, 32, 16, 16, True, True, True),      # channels-last, ten channels a group (pieces of two)
    (1, 256, 16, 16, 24, False, True, True),     # sixteen channels (pieces of four)
    (2, 240, 16, 16, 16, True, True, True),      # fifteen
    (1, 1280, 32, 8, 8, True, True, True),       # forty
    (1, 256, 2, 32, 64, True, True, True),       # eight CTAs with all the values they hold
    (1, 256, 256, 16, 16, False, True, True),    # one channel a group
]


def test_matched():
    assert "silu" in lines(build(40, 4, 16, 12, True, False, False), 2)[0]
    assert "to channels-last" in lines(build(40, 4, 20, 18, True, False, True), 1)[0]
    assert "to channels-last" not in lines(build(256, 16, 16, 24, False, True, True), 1)[0] and " channels-last" in lines(build(256, 16, 16, 24, False, True, True), 1)[0]
    assert not lines(build(40, 4, 5, 5, True, False, False), 2)          # planes that are no multiple of four
    assert not lines(build(256, 2, 32, 68, True, True, True), 1)         # groups that eight CTAs do not hold
    g = Graph()                                                          # the layernorm is read by something else, too
    n = g.layernorm(g.view(g.input(shape(BATCH, 8, 4, 4)), shape(BATCH, 2, 64)), 2, 1e-5)
    g.output(g.add(g.mul(g.view(n, shape(BATCH, 8, 4, 4)), g.constant_tensor(np.ones((1, 8, 1, 1), np.float32))), g.constant_tensor(np.ones((1, 8, 1, 1), np.float32))))
    g.output(n)
    assert not lines(g, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n,c,groups,h,w,silu,before,after", CASES)
@pytest.mark.parametrize("offset", [0.0, 100.0])
def test_values(n, c, groups, h, w, silu, before, after, offset):
    from kyanite_b200.executor import CudaExecutor
    g = build(c, groups, h, w, silu, before, after)
    assert len(lines(g, n)) == 1
    x = (rng(c).standard_normal((n, c, h, w)) + offset).astype(np.float32)
    with CudaExecutor(0, g, n, math_mode=MATH_TF32) as ex:
        got = ex.evaluate([x])
        np.testing.assert_array_equal(got[-1], ex.evaluate([x])[-1])
    read = (got[0] if before else x).astype(np.float64)      # (the convolution's own rounding is another test's)
    y = got[1 if before else 0]
    r = rng(0)
    gamma, beta = ((a + 0.3 * r.standard_normal((1, c, 1, 1))).astype(np.float32).astype(np.float64) for a in (1, 0))
    flat = read.reshape(n, groups, -1)
    want = ((flat - flat.mean(2, keepdims=True)) / np.sqrt(flat.var(2, keepdims=True) + 1e-5)).reshape(read.shape) * gamma + beta
    if silu:
        want = want / (1 + np.exp(-want))
    # f32 statistics: a mean is off by an ulp or two of the values, which next to a deviation of one is 100 x 2^-23 at the offset
    assert np.abs(y - want).max() <= (2e-5 + offset * 6e-7) * np.abs(want).max()
