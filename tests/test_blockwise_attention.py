"""Attention in one step over any number of keys (kernels/flash.cu): ragged rows and keys, an additive term, f16 storage, head
dimensions up to 128.  The reference runs the scores matmul, the scaling, the sum, the softmax and the second matmul as
operations of their own: kn-cuda-eval/src/planner.rs:300-330 and 560-600."""
import re

import numpy as np
import pytest

from kyanite_b200.configs import _attention
from kyanite_b200.executor import FLAG_NO_PERSISTENT_GEMM, MATH_F32, MATH_TF32, plan_describe
from kyanite_b200.graph import BATCH, DType, Graph, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph

SHAPES = {
    # name: (b, m, n, k, dv)
    "one_short_block": (12, 120, 120, 64, 64),
    "smallest": (2, 16, 16, 8, 8),
    "one_column_past_a_block": (3, 129, 129, 40, 40),
    "cross_attention": (4, 200, 77, 80, 80),
    "many_blocks": (2, 130, 1000, 64, 64),
    "widest_head": (2, 333, 333, 128, 128),
    "values_wider_than_head": (2, 77, 260, 32, 128),
    "more_items_than_the_chip_holds": (320, 100, 150, 64, 64),
}
# f32 goes this way only where its two matmuls by themselves would round their operands to TF32 (test_operand_rounding.py):
# at least 64 rows, and 0.2 GFLOP or V along its keys.  So there are more batch entries of each in f32.
F32_BATCH = {"one_short_block": 120, "one_column_past_a_block": 160, "cross_attention": 100, "many_blocks": 13, "widest_head": 8,
             "values_wider_than_head": 40, "more_items_than_the_chip_holds": 320}
TERMS = ["none", "input", "per_head", "causal", "lowest", "blocks_of_infinity"]
CONSTANT = ("causal", "lowest", "blocks_of_infinity")


def constant_term(kind, m, n, dtype, r):
    if kind == "causal":
        return np.triu(np.full((1, m, n), -np.inf, dtype), 1)
    if kind == "lowest":        # the lowest finite value, which absorbs the scores; one row has nothing else
        t = np.where(r.random((1, m, n)) < 0.5, np.finfo(dtype).min, 0).astype(dtype)
        t[0, 3] = np.finfo(dtype).min
        return t
    t = np.zeros((1, m, n), dtype)   # a row whose first keys are all masked, one that sees the last key only, a dead one
    t[0, 1, : max(n - 3, 1)] = -np.inf
    t[0, 2, : n - 1] = -np.inf
    t[0, 5] = -np.inf
    return t


def build(name, half, kind, seed=0):
    b, m, n, k, dv = SHAPES[name]
    if not half:
        b = F32_BATCH.get(name, b)
    dtype, np_dtype = (DType.F16, np.float16) if half else (DType.F32, np.float32)
    r = np.random.Generator(np.random.PCG64(seed))
    g = Graph()
    q, keys, v = (g.input(shape(*s), dtype) for s in ((b, m, k), (b, n, k), (b, n, dv)))
    inputs = [r.standard_normal(s).astype(np_dtype) for s in ((b, m, k), (b, n, k), (b, n, dv))]
    scores = g.mul(g.batched_mat_mul(q, g.permute(keys, [0, 2, 1])), g.scalar(1.0 / np.sqrt(k), dtype))
    if kind in ("input", "per_head"):
        s = (b if kind == "per_head" else 1, m, n)
        scores = g.add(scores, g.input(shape(*s), dtype))
        inputs.append(r.standard_normal(s).astype(np_dtype))
    elif kind != "none":
        scores = g.add(scores, g.constant_tensor(constant_term(kind, m, n, np_dtype, r)))
    g.output(g.batched_mat_mul(g.softmax(scores, 2), v))
    return g, inputs


def one_step(g, mode=MATH_TF32, flags=0):
    return [l for l in plan_describe(g, 0, mode, flags=flags).splitlines() if "blockwise-attention" in l]


@pytest.mark.parametrize("half", [False, True], ids=["f32", "f16"])
def test_route(half):
    for kind in TERMS:
        g, _ = build("widest_head", half, kind)
        lines = one_step(g)
        assert len(lines) == 1 and ("+term" in lines[0]) == (kind != "none"), lines
        assert ("by blocks" in lines[0]) == (kind in CONSTANT), lines
        assert not one_step(g, MATH_F32) and not one_step(g, flags=FLAG_NO_PERSISTENT_GEMM)


@pytest.mark.gpu
@pytest.mark.parametrize("half", [False, True], ids=["f32", "f16"])
@pytest.mark.parametrize("kind", TERMS)
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_matches_oracle(name, kind, half):
    from kyanite_b200.executor import CudaExecutor
    if name == "more_items_than_the_chip_holds" and kind not in ("none", "causal"):
        pytest.skip("the oracle takes long over it, and the smaller shapes have this term")
    if not half and name not in F32_BATCH:
        pytest.skip("too few rows: f32 operands stay f32")
    g, inputs = build(name, half, kind, seed=7)
    assert len(one_step(g)) == 1
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)
        again = ex.evaluate(inputs)
    # two chained contractions over operands of 11 bits, and in f16 the oracle's own rounding of scores up to 16 in size
    # (2^-8 apart at most, half of that in the exponent): 4e-3 of the largest magnitude
    assert_tensors_match(expected, got, 4e-3, 4e-3, abs_scaled=True)
    assert np.array_equal(got[0], again[0], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("b,s,h,d,half", [(1, 100, 3, 64, True), (3, 100, 3, 64, True), (2, 33, 4, 32, True), (1, 333, 16, 64, False),
                                          (3, 200, 32, 32, False)])
def test_heads_split_and_merged(b, s, h, d, half):
    """The head split is read in place and the heads are merged by the step's own stores."""
    from kyanite_b200.executor import CudaExecutor
    dtype = DType.F16 if half else DType.F32
    g = Graph()
    q, k, v = (g.input(shape(BATCH * s, h * d), dtype) for _ in range(3))
    g.output(_attention(g, q, k, v, s, s, h, d, BATCH, dtype=dtype))
    lines = [l for l in plan_describe(g, b, MATH_TF32).splitlines() if l.startswith("step")]
    assert len(lines) == 1 and "heads merged" in lines[0], lines
    r = np.random.Generator(np.random.PCG64(4))
    inputs = [r.standard_normal((b * s, h * d)).astype(dtype.np) for _ in range(3)]
    expected = cpu_eval_graph(g.to_bytes(), b, inputs)
    with CudaExecutor(0, g, b, math_mode=MATH_TF32) as ex:
        assert_tensors_match(expected, ex.evaluate(inputs), 4e-3, 4e-3, abs_scaled=True)


@pytest.mark.gpu
@pytest.mark.parametrize("half", [False, True], ids=["f32", "f16"])
def test_not_finite_behind_the_mask(half):
    """Blocks that a causal mask hides are left out only where they would add exact zeros: a NaN or an infinity in a hidden key
    or value reaches the rows that do not see it, as -infinity + infinity and 0 * infinity are NaN."""
    from kyanite_b200.executor import CudaExecutor
    b, s, d = 80, 300, 32
    dtype = DType.F16 if half else DType.F32
    r = np.random.Generator(np.random.PCG64(11))
    g = Graph()
    q, keys, v = (g.input(shape(b, s, d), dtype) for _ in range(3))
    scores = g.add(g.mul(g.batched_mat_mul(q, g.permute(keys, [0, 2, 1])), g.scalar(0.2, dtype)), g.constant_tensor(constant_term("causal", s, s, dtype.np, r)))
    g.output(g.batched_mat_mul(g.softmax(scores, 2), v))
    assert "masked ones left out" in one_step(g)[0]
    inputs = [r.standard_normal((b, s, d)).astype(dtype.np) for _ in range(3)]
    inputs[1][7, 290, 0], inputs[1][20, 150, 3], inputs[1][33, 299, 1] = np.inf, -np.inf, np.nan
    inputs[2][3, 299, 5], inputs[2][11, 200, 7], inputs[2][12, 130, 31] = np.nan, np.inf, -np.inf
    with np.errstate(all="ignore"):
        expected = cpu_eval_graph(g.to_bytes(), 0, inputs)[0]
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)[0]
    assert 1000 < np.isnan(expected).sum() < expected.size / 10
    np.testing.assert_array_equal(np.isnan(got), np.isnan(expected))
    infinite, finite = np.isinf(expected), np.isfinite(expected)
    np.testing.assert_array_equal(got[infinite], expected[infinite])
    assert_tensors_match([expected[finite]], [got[finite]], 4e-3, 4e-3, abs_scaled=True)


def test_a_mask_is_prepared_once():
    """The layers of a decoder share one mask: its padded form and its table by blocks are made once and read by all."""
    s, d = 333, 32
    r = np.random.Generator(np.random.PCG64(1))
    g = Graph()
    mask = g.constant_tensor(constant_term("causal", s, s, np.float16, r))
    for heads in (2, 2, 5):
        q, keys, v = (g.input(shape(heads, s, d), DType.F16) for _ in range(3))
        g.output(g.batched_mat_mul(g.softmax(g.add(g.batched_mat_mul(q, g.permute(keys, [0, 2, 1])), mask), 2), v))
    lines = one_step(g)
    prepared = {tuple(re.findall(r"r:\w+@(b\d+)", line)[-2:]) for line in lines}
    assert len(lines) == 3 and len(prepared) == 1, lines
    const_bytes = int(re.search(r"const_bytes=(\d+)", plan_describe(g, 0, MATH_TF32)).group(1))
    assert const_bytes < 2 * s * (s + 384) + 4096     # the mask, its rows padded to 384, the table
