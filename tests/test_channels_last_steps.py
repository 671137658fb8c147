"""Concatenations, enlargements and elementwise steps between channels-last convolutions: where the planner keeps their results
channels-last, that it falls back to plain memory elsewhere, and that the values are the oracle's either way."""
import numpy as np
import pytest

from kyanite_b200.executor import MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, Graph, UnaryOp, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph


def rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def conv(g, t, cin, cout, seed, size=3):
    w = (rng(seed).standard_normal((cout, cin, size, size)) / np.sqrt(size * size * cin)).astype(np.float32)
    return g.conv(t, g.constant_tensor(w), 1, 1, size // 2, size // 2)


def enlarge(g, t, c, h, w):
    """nearest neighbour, twice the height, then twice the width"""
    t = g.view(g.broadcast(g.view(t, shape(BATCH, c, h, 1, w)), shape(BATCH, c, h, 2, w)), shape(BATCH, c, 2 * h, w))
    return g.view(g.broadcast(g.view(t, shape(BATCH, c, 2 * h, w, 1)), shape(BATCH, c, 2 * h, w, 2)), shape(BATCH, c, 2 * h, 2 * w))


def build(name):
    g = Graph()
    c, h, w = 256, 8, 16
    x = g.input(shape(BATCH, c, h, w))
    a = conv(g, x, c, c, 1)                    # channels-last where a convolution reads it too
    b = conv(g, a, c, c, 2)
    if name == "concat":                       # of two such results, read by a third convolution
        g.output(conv(g, b, c, 64, 4))
        y = conv(g, g.concat([a, b], 1), 2 * c, 64, 3)
    elif name == "concat_with_plain":          # one part lies as the caller gave it
        g.output(b)
        y = conv(g, g.concat([a, x], 1), 2 * c, 64, 3)
    elif name == "concat_of_sums":             # elementwise steps over channels-last parts
        g.output(conv(g, b, c, 64, 4))
        y = conv(g, g.concat([g.unary(UnaryOp.TANH, g.mul(a, b)), b], 1), 2 * c, 64, 3)
    elif name == "enlarged":
        y = conv(g, enlarge(g, b, c, h, w), c, 64, 3)
    elif name == "enlarged_twice_read":        # also by something that wants plain memory
        e = enlarge(g, a, c, h, w)
        g.output(g.softmax(g.view(e, shape(BATCH, c * 4, h * w)), 2))
        y = conv(g, e, c, 64, 3)
    elif name == "flattened":                  # a view that channels-last memory cannot express
        g.output(b)
        y = g.softmax(g.view(a, shape(BATCH, c * h * w)), 1)
    elif name == "concat_along_rows":
        g.output(conv(g, b, c, 64, 4))
        y = conv(g, g.concat([a, b], 2), c, 64, 3)
    else:                                      # channels that are no multiple of four
        d = conv(g, b, c, 30, 4)
        g.output(conv(g, d, 30, 64, 5))
        y = conv(g, g.concat([d, a], 1), c + 30, 64, 3)
    g.output(y)
    return g


NAMES = ["concat", "concat_with_plain", "concat_of_sums", "enlarged", "enlarged_twice_read", "flattened", "concat_along_rows", "odd_channels"]


def test_no_turning_copies():
    """The copies of an enlargement and of a concatenation move whole rows of channels."""
    for name in ("concat", "enlarged"):
        lines = [l for l in plan_describe(build(name), 2, MATH_TF32).splitlines() if l.startswith("step") and " copy " in l]
        assert len([l for l in lines if " vec4 acc" in l]) == 2, lines


def group_norm(g, t, c, groups, h, w, scale=True):
    y = g.view(g.layernorm(g.view(t, shape(BATCH, groups, c // groups * h * w)), 2, 1e-5), shape(BATCH, c, h, w))
    one = lambda: g.constant_tensor(np.ones((1, c, 1, 1), np.float32))  # noqa: E731
    return g.add(g.mul(y, one()), one()) if scale else g.add(y, one())


@pytest.mark.parametrize("h,w,scale,view", [(9, 10, True, False), (16, 16, False, False), (16, 16, True, True), (7, 7, False, True)])
def test_convolutions_before_a_norm_that_reads_plain_memory(h, w, scale, view):
    """Planes that are no multiple of four, a norm without a scale, a result that is viewed: no copy between convolution and norm."""
    c, g = 64, Graph()
    x = conv(g, g.input(shape(BATCH, c, h, w)), c, c, 1)
    g.output(g.unary(UnaryOp.TANH, x))
    y = group_norm(g, x, c, 16, h, w, scale)
    g.output(conv(g, y, c, c, 2))
    if view:
        g.output(g.view(y, shape(BATCH, c, h * w)))
    lines = [l.split()[2] for l in plan_describe(g, 4, MATH_TF32).splitlines() if l.startswith("step")]
    # the input turned, the convolution, its tanh, the norm [and its scale and shift], turned for the second convolution
    assert lines.count("Scalar") == (4 if "Layernorm" in lines else 3 if view else 2), lines


def test_copies_that_nobody_wants_channels_last():
    """Concatenated and enlarged images that a softmax, a plain norm or the caller reads are written in plain memory at once."""
    c, h, w, g = 256, 8, 16, Graph()
    x = g.input(shape(BATCH, c, h, w))
    a = conv(g, x, c, c, 1)
    b = conv(g, a, c, c, 2)                    # (channels-last, both)
    g.output(conv(g, b, c, 64, 3))
    g.output(g.concat([a, b], 1))
    g.output(enlarge(g, a, c, h, w))
    copies = [l for l in plan_describe(g, 2, MATH_TF32).splitlines() if l.startswith("step") and " copy " in l]
    assert len(copies) == 1 + 2 + 2, copies    # the input, the two parts, two enlargements


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("name", NAMES)
def test_values(name, batch):
    from kyanite_b200.executor import CudaExecutor
    g = build(name)
    x = rng(5).standard_normal((batch, 256, 8, 16)).astype(np.float32)
    expected = cpu_eval_graph(g.to_bytes(), batch, [x])
    with CudaExecutor(0, g, batch, math_mode=MATH_TF32) as ex:
        # two contractions of TF32 operands in a row
        assert_tensors_match(expected, ex.evaluate([x]), 4e-3, 4e-3, abs_scaled=True)
