"""Matmuls of less than one round of the chip: one tile and one K slice per CTA, the slices of a tile summed inside a cluster
(gemm_slices_kernel).  The reference calls cublasSgemmStridedBatched and a kernel for what follows:
kn-cuda-sys/src/wrapper/group.rs:120-171."""
import re

import numpy as np
import pytest

from kyanite_b200._lib import KN_FLAG_TRACE_GEMM
from kyanite_b200.executor import FLAG_NO_PERSISTENT_GEMM, MATH_F32, MATH_TF32, plan_describe
from kyanite_b200.graph import DType, Graph, shape
from oracle.cpu_eval import assert_tensors_match, cpu_eval_graph

SHAPES = [
    # (b, m, n, k)
    (1, 64, 16, 512),        # one tile, narrower than its 32 columns
    (1, 120, 768, 768),
    (1, 129, 100, 1000),     # a row past a tile, a ragged last column block, a K tail
    (1, 333, 200, 96),       # fewer K blocks than a cluster has CTAs
    (3, 100, 72, 260),
    (1, 256, 1024, 4096),
    (2, 128, 33 * 4, 2048),
]


def build(b, m, n, k, half=False, bias=False, residual=False, relu=False, constant=True, seed=0):
    r = np.random.Generator(np.random.PCG64(seed))
    dtype, np_dtype = (DType.F16, np.float16) if half else (DType.F32, np.float32)
    g = Graph()
    x = g.input(shape(b, m, k), dtype)
    inputs = [r.standard_normal((b, m, k)).astype(np_dtype)]
    weights = (r.standard_normal((b, n, k)) / np.sqrt(k)).astype(np_dtype)
    if constant:
        w = g.constant_tensor(weights)
    else:
        w = g.input(shape(b, n, k), dtype)
        inputs.append(weights)
    y = g.batched_mat_mul(x, g.permute(w, [0, 2, 1]))
    if bias:
        y = g.add(y, g.constant_tensor(r.standard_normal((1, 1, n)).astype(np_dtype)))
    if residual:
        y = g.add(y, g.input(shape(b, m, n), dtype))
        inputs.append(r.standard_normal((b, m, n)).astype(np_dtype))
    if relu:
        y = g.relu(y)
    g.output(y)
    return g, inputs


def tile(g, mode=MATH_TF32, flags=0):
    lines = [l for l in plan_describe(g, 0, mode, flags=flags).splitlines() if " tile=" in l]
    return lines[0] if lines else ""


def test_rule():
    for b, m, n, k in SHAPES:
        line = tile(build(b, m, n, k)[0])
        assert line, (b, m, n, k)
        slices = re.search(r"splitk=(\d+) in a cluster", line)
        width = int(re.search(r"tile=(\d+)", line).group(1))
        assert width % 32 == 0 and 32 <= width <= 256 and width - 32 < n
        assert slices is None or 2 <= int(slices.group(1)) <= min(8, -(-k // 32)), line
        assert not tile(build(b, m, n, k)[0], MATH_F32) and not tile(build(b, m, n, k)[0], flags=FLAG_NO_PERSISTENT_GEMM)
        assert not tile(build(b, m, n, k)[0], flags=KN_FLAG_TRACE_GEMM)   # its markers are the persistent kernel's
    assert not tile(build(1, 4096, 4096, 512)[0])     # rounds of wide tiles: the persistent kernel


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["plain", "bias_relu", "bias_residual", "both_inputs", "f16"])
@pytest.mark.parametrize("b,m,n,k", SHAPES)
def test_matches_oracle(b, m, n, k, what):
    from kyanite_b200.executor import CudaExecutor
    half = what == "f16"
    if half and (k % 8 != 0 or n % 8 != 0):
        pytest.skip("rows of f16 that are no multiple of 16 bytes are copied or computed elsewhere")
    g, inputs = build(b, m, n, k, half, bias="bias" in what, residual="residual" in what, relu="relu" in what,
                      constant=what != "both_inputs", seed=3)
    assert tile(g)
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)
        again = ex.evaluate(inputs)
    # products of operands of 11 bits (TF32, f16), f32 sums; results of size 1: 2e-3 of the largest
    assert_tensors_match(expected, got, 2e-3, 2e-3, abs_scaled=True)
    assert np.array_equal(got[0], again[0])


@pytest.mark.gpu
def test_behind_a_long_kernel():
    """What runs in front of it does not count towards the limit of its waits: a reduction of seconds, then a sliced matmul,
    which is resident from that kernel's start on."""
    from kyanite_b200.executor import CudaExecutor
    alone, inputs = build(1, 120, 96, 512, seed=4)
    expected = cpu_eval_graph(alone.to_bytes(), 0, inputs)
    r = np.random.Generator(np.random.PCG64(4))
    g = Graph()
    k = 1 << 28
    row = g.broadcast(g.view(g.input(shape(1), DType.F16), shape(1, 1, 1)), shape(1, 1, k))   # (reads one element k times)
    g.output(g.batched_mat_mul(row, g.permute(row, [0, 2, 1])))
    x = g.input(shape(1, 120, 512))
    r.standard_normal((1, 120, 512))
    w = g.constant_tensor((r.standard_normal((1, 96, 512)) / np.sqrt(512)).astype(np.float32))
    g.output(g.batched_mat_mul(x, g.permute(w, [0, 2, 1])))
    steps = [l for l in plan_describe(g, 0, MATH_TF32).splitlines() if l.startswith("step")]
    assert len(steps) == 2 and " tile=" in steps[1], steps
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate([np.ones(1, np.float16), inputs[0]])
    assert_tensors_match(expected, got[1:], 2e-3, 2e-3, abs_scaled=True)


# the ways an addend reaches the rows: shared by all, one value per row, one per element, along the rows instead of the columns
@pytest.mark.gpu
@pytest.mark.parametrize("b,m,n,k", [(1, 129, 96, 64), (1, 250, 320, 1280), (2, 100, 132, 768), (1, 120, 96, 4096)])
@pytest.mark.parametrize("kinds", ["row", "row_element", "element_column", "element_element", "across", "row_across"])
def test_addends(b, m, n, k, kinds):
    from kyanite_b200.executor import CudaExecutor
    r = np.random.Generator(np.random.PCG64(m + n))
    g = Graph()
    y = g.batched_mat_mul(g.input(shape(b, m, k)), g.permute(g.constant_tensor((r.standard_normal((b, n, k)) / np.sqrt(k)).astype(np.float32)), [0, 2, 1]))
    inputs = [r.standard_normal((b, m, k)).astype(np.float32)]
    for kind in kinds.split("_"):
        if kind in ("row", "column"):
            y = g.add(y, g.constant_tensor(r.standard_normal((b, m, 1) if kind == "row" else (b, 1, n)).astype(np.float32)))
        else:
            s = (b, n, m) if kind == "across" else (b, m, n)
            t = g.input(shape(*s))
            inputs.append(r.standard_normal(s).astype(np.float32))
            y = g.add(y, g.permute(t, [0, 2, 1]) if kind == "across" else t)
    g.output(y)
    assert tile(g)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        got = ex.evaluate(inputs)
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)
    # k products of operands rounded to 11 bits, each off by 2^-11 of itself: a sum of size 1 is off by 2^-11, five times that covers the largest of them
    assert np.abs(got[0].astype(np.float64) - expected[0]).max() <= 5 * 2.0 ** -11 * max(1.0, np.abs(expected[0]).max() / 3)


# how many slices the planner takes, and with it which of the kernel's row loops runs (1, 2, up to 4, up to 8)
COUNTS = [
    # (half, b, m, n, k, slices)
    (False, 1, 250, 320, 96, 1), (False, 1, 129, 2304, 768, 2), (False, 3, 190, 768, 768, 2), (False, 1, 250, 1280, 768, 3),
    (False, 1, 120, 1000, 520, 4), (False, 1, 129, 768, 768, 5), (False, 1, 120, 384, 768, 8),
    (True, 1, 129, 2304, 2048, 2), (True, 1, 333, 768, 1280, 3), (True, 1, 120, 1000, 1280, 4), (True, 1, 129, 136, 1280, 7),
]


def count(g):
    slices = re.search(r"splitk=(\d+) in a cluster", tile(g))
    return int(slices.group(1)) if slices else 1


@pytest.mark.parametrize("half,b,m,n,k,slices", COUNTS)
def test_slice_counts(half, b, m, n, k, slices):
    assert count(build(b, m, n, k, half)[0]) == slices


@pytest.mark.gpu
@pytest.mark.parametrize("half,b,m,n,k,slices", [c for c in COUNTS if c[0]])
def test_slice_counts_f16(half, b, m, n, k, slices):
    """(a sum or an activation of f16 values rounds once more and is a step of its own)"""
    from kyanite_b200.executor import CudaExecutor
    g, inputs = build(b, m, n, k, half, seed=n)
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        assert_tensors_match(expected, ex.evaluate(inputs), 2e-3, 2e-3, abs_scaled=True)   # (as in test_matches_oracle)


@pytest.mark.gpu
@pytest.mark.parametrize("act", ["none", "relu", "gelu"])
@pytest.mark.parametrize("elements", [0, 1, 2])
@pytest.mark.parametrize("half,b,m,n,k,slices", [c for c in COUNTS if not c[0]])
def test_row_loops(half, b, m, n, k, slices, elements, act):
    """Every number of slices with no, one and two addends that differ by row (with one of them, a bias too)."""
    from kyanite_b200.configs import _gelu
    from kyanite_b200.executor import CudaExecutor
    r = np.random.Generator(np.random.PCG64(n + elements))
    g, inputs = build(b, m, n, k, bias=elements == 1, seed=n)
    y = g.outputs.pop()
    for _ in range(elements):
        y = g.add(y, g.input(shape(b, m, n)))
        inputs.append(r.standard_normal((b, m, n)).astype(np.float32))
    y = {"none": lambda: y, "relu": lambda: g.relu(y), "gelu": lambda: _gelu(g, y)}[act]()
    g.output(y)
    assert count(g) == slices and len([l for l in plan_describe(g, 0, MATH_TF32).splitlines() if l.startswith("step")]) == 1
    expected = cpu_eval_graph(g.to_bytes(), 0, inputs)
    with CudaExecutor(0, g, 0, math_mode=MATH_TF32) as ex:
        assert_tensors_match(expected, ex.evaluate(inputs), 2e-3, 2e-3, abs_scaled=True)   # (as in test_matches_oracle)
