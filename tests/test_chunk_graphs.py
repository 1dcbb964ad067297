"""Runs that go through the chunk graph, against single steps: the same bits. A
run of a few steps instantiates the step graph, one that reaches the chunk graph
a second one, which is how these tests know that they reached it."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

SIZES = (20_000, 300, 8193)  # one alone, or a mixed table of the separate kernels


def run(native, sizes, parts, chunk=10):
    """States after the parts' steps, and the graphs instantiated."""
    with native.Batch() as b:
        b.tune(graph_chunk=chunk)
        ids = [b.add(native.generate(n, n)) for n in sizes]
        for k in parts:
            b.step(k)
        return [b.read(i) for i in ids], b.graph_counts()[0]


def same(a, b):
    return all(t == u and x.tobytes() == y.tobytes() for (t, x), (u, y) in zip(a, b))


@pytest.mark.parametrize("flocks", [1, 3])
@pytest.mark.parametrize("chunk, parts", [(10, (123,)), (10, (10,) * 6), (4, (40, 3, 8)), (7, (7, 9, 7, 15, 14))])
def test_chunks_equal_single_steps(native, flocks, chunk, parts):
    got, graphs = run(native, SIZES[:flocks], parts, chunk)
    want, none = run(native, SIZES[:flocks], (1,) * sum(parts))
    assert graphs == 2 and none == 0
    assert same(got, want)


def test_flocks_that_stop_join_and_leave_between_chunks(native):
    plan = [(0, 115), (1, 33), (2, 101)]  # flocks that stop within a chunk
    with native.Batch() as b:
        ids = [b.add(native.generate(n, n)) for n in SIZES]
        b.step_each([ids[k] for k, _ in plan], [s for _, s in plan])
        for _ in range(5):
            b.step(10)
        late = b.add(native.generate(9000, 1))  # other sizes: the graphs are captured again
        for _ in range(5):
            b.step(10)
        b.remove(ids[1])
        b.step(120)
        inst, updated = b.graph_counts()
        assert inst == 2 and updated >= 3
        for i, n, seed, steps in ((ids[0], SIZES[0], SIZES[0], 335), (ids[2], SIZES[2], SIZES[2], 321),
                                  (late, 9000, 1, 170)):
            with native.Batch() as a:
                k = a.add(native.generate(n, seed))
                for _ in range(steps):
                    a.step(1)
                assert same([b.read(i)], [a.read(k)])
