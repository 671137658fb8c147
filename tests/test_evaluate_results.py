"""Results of `evaluate` belong to the caller: whatever later evaluations do, and beyond the executor's life, for results
that are handed out as pinned memory (64 KB and more), for small ones and when more are kept than there are sets."""
import numpy as np
import pytest

from kyanite_b200.executor import CudaExecutor
from kyanite_b200.graph import BATCH, Graph, SliceRange, shape

pytestmark = pytest.mark.gpu


# columns on either side of the limits of the transfer kernel and of handing results out; enough input for staged uploads
@pytest.mark.parametrize("columns", [3, 16384, 16388, 300001])
def test_results_are_the_callers(columns):
    g = Graph()
    x = g.input(shape(BATCH, columns))
    g.output_all([g.add(x, g.scalar(1.0)), g.mul(x, g.scalar(2.0))])
    rng = np.random.default_rng(columns)
    inputs = [rng.standard_normal((1, columns)).astype(np.float32) for _ in range(9)]
    with CudaExecutor(0, g, 1) as ex:
        kept = [ex.evaluate([a]) for a in inputs]          # more than an executor has sets
        del kept[3]
        again = ex.evaluate([inputs[3]])                   # a returned set serves again
        ex.evaluate_begin([inputs[0]])
        staged = [a.copy() for a in ex.evaluate_end()]
    kept.insert(3, again)
    kept.append(staged)
    for a, (plus, twice) in zip(inputs + [inputs[0]], kept):
        np.testing.assert_array_equal(plus, a + np.float32(1))
        np.testing.assert_array_equal(twice, a * np.float32(2))
        plus[...] = 0                                      # and they are writable


def test_waits_for_the_callers_own_transfers():
    """A caller that has the stream may copy from the staging buffers on it; `evaluate` stages new inputs after that."""
    import torch
    g = Graph()
    g.output(g.add(g.input(shape(1, 1000)), g.scalar(1.0)))
    with CudaExecutor(0, g, 1) as ex:
        ex.evaluate([np.zeros((1, 1000), np.float32)])
        stream = torch.cuda.ExternalStream(ex.stream())
        ex.host_inputs[0][...] = 7
        taken = torch.empty(1, 1000, device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(50_000_000)   # some 25 ms
            taken.copy_(torch.from_numpy(ex.host_inputs[0]), non_blocking=True)
        ex.evaluate([np.zeros((1, 1000), np.float32)])
        stream.synchronize()
        assert (taken == 7).all()


def test_results_too_large_to_pin():
    g = Graph()
    x = g.input(shape(1, 1))
    g.output(g.add(g.broadcast(x, shape(1, 33 << 20)), g.scalar(1.0)))     # 132 MB
    with CudaExecutor(0, g, 0) as ex:
        got, = ex.evaluate([np.full((1, 1), 4, np.float32)])
    assert got.flags.owndata and (got == 5).all()


def test_no_later_evaluation_prepares_results():
    """The first evaluation makes all the sets of pinned results and the graphs that download into them: whatever the ones after
    it hold, no other pinned memory appears."""
    g = Graph()
    x = g.input(shape(BATCH, 100000))
    g.output(g.add(x, g.scalar(1.0)))
    a = np.arange(100000, dtype=np.float32).reshape(1, -1)
    with CudaExecutor(0, g, 1) as ex:
        kept, addresses = [], set()
        for _ in range(9):
            del kept[:-3]                       # three held, the fourth set free
            kept.append(ex.evaluate([a])[0])
            assert not kept[-1].flags.owndata
            addresses.update(r.ctypes.data for r in kept)
        assert len(addresses) == 4
        more = [ex.evaluate([a])[0], ex.evaluate([a])[0]]   # all sets held: arrays of their own
        assert all(r.flags.owndata for r in more)
        for r in kept + more:
            np.testing.assert_array_equal(r, a + np.float32(1))


def test_small_results_do_not_hold_large_ones():
    """A small result is an array of its own: one that is kept does not keep the memory of the large one beside it, and later
    evaluations go on being handed out without a copy."""
    g = Graph()
    x = g.input(shape(BATCH, 40000))
    g.output_all([g.mul(x, g.scalar(2.0)), g.add(g.slice(x, 1, SliceRange(0, 5)), g.scalar(1.0))])
    rng = np.random.default_rng(1)
    inputs = [rng.standard_normal((1, 40000)).astype(np.float32) for _ in range(6)]
    with CudaExecutor(0, g, 1) as ex:
        small, addresses = [], set()
        for a in inputs:
            large, few = ex.evaluate([a])
            np.testing.assert_array_equal(large, a * np.float32(2))
            assert few.flags.owndata and not large.flags.owndata
            addresses.add(large.ctypes.data)
            small.append(few)
            del large
    for a, few in zip(inputs, small):
        np.testing.assert_array_equal(few, a[:, :5] + np.float32(1))
    assert len(addresses) <= 4


def test_executors_of_several_threads():
    """Executors of their own, evaluated at once: large inputs and results find the copy helpers taken or free."""
    import threading
    g = Graph()
    g.output(g.add(g.input(shape(BATCH, 300001)), g.scalar(1.0)))
    failures = []

    def user(seed):
        rng = np.random.default_rng(seed)
        kept = []
        try:
            with CudaExecutor(0, g, 2) as ex:
                for _ in range(12):
                    a = rng.standard_normal((2, 300001)).astype(np.float32)
                    kept.append((a, ex.evaluate([a])[0]))
                    kept = kept[-4:]
                    for a, got in kept:
                        np.testing.assert_array_equal(got, a + np.float32(1))
        except BaseException as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=user, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
