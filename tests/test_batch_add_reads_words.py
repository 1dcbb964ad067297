"""Batch.add has read its array when it returns, whatever memory that is: the
caller may change it at once, and the memory of a dropped one may be handed out
again. Bit-exact: the words are moved, not computed with."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 400_000  # 24 MB: a copy of about 0.1 ms on the link


def test_arrays_straight_from_read(native):
    # each temporary dies with its add, and the next read() gets its block
    flocks = [native.Flock(native.generate(N - k, 1 + k)) for k in range(6)]
    with native.Batch() as b:
        ids = [b.add(f.read()[1]) for f in flocks]
        for f, i in zip(flocks, ids):
            assert b.read(i)[1].tobytes() == f.read()[1].tobytes()
    for f in flocks:
        f.close()


@pytest.mark.parametrize("locked", [False, True])
def test_an_array_changed_after_each_add(native, locked):
    with native.Flock(native.generate(N, 5)) as f:
        w = f.read()[1]  # page-locked
    if not locked:
        w = w.copy()
    with native.Batch() as b:
        ids, want = [], []
        for k in range(6):
            ids.append(b.add(w))
            want.append(w.tobytes())
            w[:, 0] += np.float32(1.0)
        for i, x in zip(ids, want):
            assert b.read(i)[1].tobytes() == x
