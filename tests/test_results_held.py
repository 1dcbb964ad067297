"""A program that keeps its results locks no more than 2 GiB of host memory: the
results beyond that are ordinary arrays with the same words."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

N = 1_000_000  # a 60 MB result, a block of 64 MB (or less)


def test_results_are_page_locked_up_to_two_gib(native):
    straight = native.lib().flk_copies_straight
    with native.Flock(native.generate(N, 1)) as f:
        want = f.read()[1].tobytes()
        held = [f.read()[1] for _ in range(38)]
        locked = [bool(straight(w.ctypes.data, w.nbytes)) for w in held]
        count = sum(locked)
        assert (2 << 30) // (64 << 20) <= count <= (2 << 30) // (N * 60) < len(held)
        assert locked == [True] * count + [False] * (len(held) - count)
        assert all(w.tobytes() == want for w in (held[0], held[count - 1], held[count], held[-1]))
        del held[count - 1]
        w = f.read()[1]  # the block that came back
        assert straight(w.ctypes.data, w.nbytes) == 1 and w.tobytes() == want
