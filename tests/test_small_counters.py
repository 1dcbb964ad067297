"""The work counters of long runs of small flocks: the kernel that runs all their
steps counts in 32 bits, the totals are 64-bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_counters_of_a_long_run(native):
    # every bird decides in every step (its next decision lies far behind) and has
    # every bird as a candidate (no box bounds a radius that is no number): 2^16
    # tests per warp and step, 2^32 after 65,536 steps
    n, steps = 4096, 66_000
    w = native.generate(n, 1)
    w[:, 8] = np.nan
    w[:, 12] = -1e6
    with native.Flock(w) as f:
        f.step(steps)
        assert f.counters() == (steps * n, steps * n * n, 0)


def test_a_run_of_several_launches(native):
    # a launch holds 8,192 steps; the state is what the same steps in other parts give
    w = native.generate(300, 3)
    with native.Flock(w) as f, native.Flock(w) as g:
        f.step(16_400)
        for k in (1, 8191, 5, 8203):
            g.step(k)
        assert f.counters() == g.counters()
        (t, x), (u, y) = f.read(), g.read()
    assert t == u and x.tobytes() == y.tobytes()
