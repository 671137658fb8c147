"""Elementwise programs over vectors at the sizes from which a thread takes two and four positions (elementwise.cu, launch_scalar),
with a last block that is not full, against the oracle."""
import numpy as np
import pytest

from kyanite_b200.executor import CudaExecutor, plan_describe
from kyanite_b200.graph import DType, Graph, shape
from oracle.cpu_eval import cpu_eval_graph

F16, F32 = DType.F16, DType.F32


# without a row added: tensors read as one row, of which four positions a thread are taken from 1.52 M to 2.42 M and from 4.25 M on
ONE_ROW = [(F32, F32, 1457, 1040), (F32, F32, 1459, 1040), (F32, F32, 2331, 1040), (F32, F32, 2333, 1040), (F32, F32, 4093, 1040), (F16, F32, 1459, 1040),
           (F16, F32, 2333, 1040)]


def graph(a_type, b_type, rows, cols, row=True):
    """(a + b) * (a - b) [+ row]: one value waits in a register slot while the other is computed.  Of two types: in f32, rounded to
    f16 at the end."""
    g = Graph()
    a, b = g.input(shape(rows, cols), a_type), g.input(shape(rows, cols), b_type)
    if a_type != b_type:
        a = g.value_cast(a, b_type)
    y = g.mul(g.add(a, b), g.sub(a, b))
    if row:
        y = g.add(y, g.input(shape(1, cols), b_type))
    g.output(g.value_cast(y, F16) if a_type != b_type else y)
    return g


CASES = [
    (F16, F16, 1183, 8224),   # four positions of eight halves a thread, from 9.7 M elements on
    (F16, F16, 1201, 2064),   # two, from 2.4 M on
    (F16, F16, 593, 4112),    # two where the extent would allow four
    (F16, F16, 67, 1032),     # one: rows of an odd number of positions
    (F32, F32, 4673, 1040),   # four positions of four floats, from 4.85 M elements on
    (F32, F32, 697, 1048),    # two, from 0.73 M on
    (F32, F32, 301, 1048), (F32, F32, 577, 1048),   # and from 0.3 M to 0.6 M
    (F32, F32, 587, 1048), (F32, F32, 61, 1044),    # one
    (F16, F32, 4673, 1040),   # of both types: four from 4.85 M on, else two
    (F16, F32, 697, 1048),
]


SIZES = [(*c, True) for c in CASES] + [(*c, False) for c in ONE_ROW]


@pytest.mark.parametrize("a_type,b_type,rows,cols,row", SIZES)
def test_one_program(a_type, b_type, rows, cols, row):
    steps = [line for line in plan_describe(graph(a_type, b_type, rows, cols, row), 0).splitlines() if line.startswith("step")]
    assert len(steps) == 1 and " acc" in steps[0] and (" half2" in steps[0]) == (b_type == F16), steps


@pytest.mark.gpu
@pytest.mark.parametrize("a_type,b_type,rows,cols,row", SIZES)
def test_bit_exact(a_type, b_type, rows, cols, row):
    """Every operation rounds its exact result once, in the kernel and in the oracle (which rounds f16 results by way of f32:
    innocuous for sums and products of halves)."""
    r = np.random.default_rng(rows)
    inputs = [r.standard_normal(s).astype(t.np) for s, t in (((rows, cols), a_type), ((rows, cols), b_type), ((1, cols), b_type))][:2 + row]
    g = graph(a_type, b_type, rows, cols, row)
    expected, = cpu_eval_graph(g.to_bytes(), 0, inputs)
    with CudaExecutor(0, g, 0) as ex:
        got, = ex.evaluate(inputs)
    np.testing.assert_array_equal(got, expected)
