"""States at addresses that are no multiple of four, in pageable and page-locked
memory: every word arrives and comes back. Bit-exact."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 8193])
@pytest.mark.parametrize("off", [1, 2, 3, 129])
@pytest.mark.parametrize("locked", [False, True])
def test_round_trip(native, n, off, locked):
    words = native.generate(n, n)
    raw = [np.zeros(n * 60 + 256, dtype=np.uint8) for _ in range(2)]
    k = [(-r.ctypes.data) % 64 + off for r in raw]
    w, out = (np.frombuffer(r, "<f4", n * 15, offset=o).reshape(n, 15) for r, o in zip(raw, k))
    w[:] = words
    assert w.ctypes.data % 4 == out.ctypes.data % 4 == off % 4
    with native.pinned(*(raw if locked else [])):
        with native.Flock(w) as f, native.Batch() as b:
            i = b.add(w)
            assert f.read(out)[1].tobytes() == words.tobytes()
            assert b.read(i)[1].tobytes() == words.tobytes()
    assert not raw[1][:k[1]].any() and not raw[1][k[1] + n * 60:].any()  # nothing beside the array
