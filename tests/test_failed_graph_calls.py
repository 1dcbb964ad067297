"""Runs whose graph calls fail on the host: a refused capture costs no step, a
refused launch ends the run between two steps, and the flock goes on from there.
The same bits as a flock whose calls all succeed."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 20_000


def after(native, steps):
    with native.Flock(native.generate(N, 4)) as f:
        for _ in range(steps):
            f.step(1)
        return f.read()


@pytest.mark.parametrize("runs", [(12,), (5, 7), (120,), (30, 30, 30, 30)])
def test_steps_without_graphs(native, runs):
    want = after(native, sum(runs))
    with native.Flock(native.generate(N, 4)) as f:
        f.debug_fail_graphs(captures=1000)
        for k in runs:
            f.step(k)
        t, w = f.read()
    assert t == want[0] and w.tobytes() == want[1].tobytes()


@pytest.mark.parametrize("launch", [1, 3])
@pytest.mark.parametrize("then", ["step", "debug", "retuned"])
def test_a_run_that_ends_early(native, launch, then):
    with native.Flock(native.generate(N, 4)) as f:
        f.debug_fail_graphs(launch=launch)
        with pytest.raises(native.FlockError):
            f.step(9)
        t, w = f.read()
        done = round(t / 0.005)
        want = after(native, done)
        assert 0 < done < 9 and t == want[0] and w.tobytes() == want[1].tobytes()
        if then == "debug":  # its grid is the state's own: a stale histogram would show
            d = f.step_debug()
            assert np.array_equal(np.sort(d["sorted"]), np.arange(N, dtype=np.uint32))
            with native.Flock(want[1], want[0]) as g:
                e = g.step_debug()
            assert all(np.array_equal(d[k], e[k]) for k in ("keys", "offsets", "sorted", "sets"))
            return
        if then != "step":
            f.tune_cell(3.5)  # other buckets of the same histogram
            f.tune_cell(4.0)
        f.step(7)
        got = f.read()
    want = after(native, done + 7)
    assert got[0] == want[0] and got[1].tobytes() == want[1].tobytes()
