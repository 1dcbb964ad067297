"""Snapshots asked for while their request finishes: the input, a boundary's state or
the result, whichever it is in, never a failure."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk, steps", [(1, 2), (2, 5), (5, 10)])
def test_any_moment_gives_a_state(native, chunk, steps):
    n = 700
    w = native.generate(n, 6)
    states = [w.tobytes()]
    with native.Flock(w) as f:
        for _ in range(steps):
            f.step(1)
            states.append(f.read()[1].tobytes())
    spin = np.random.default_rng(1)
    with native.Pool(1 << 30, chunk_steps=chunk) as p:
        for _ in range(400):
            ticket = p.submit(w, steps)
            seen = 0
            while p.poll(ticket) != 2:  # snapshots at every boundary, and at its end
                _, got, done = p.snapshot(ticket)
                assert seen <= done <= steps and got.tobytes() == states[done]
                seen = done
                for _ in range(int(spin.integers(0, 60))):
                    pass
            assert p.wait(ticket)[1].tobytes() == states[steps]
