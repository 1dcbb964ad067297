"""Which host memory the state kernels access directly: whole ranges of one
page-locking only. Host-side queries; no kernel touches the memory asked about."""
from __future__ import annotations

import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = mmap.PAGESIZE


def test_only_whole_page_locked_ranges(native):
    f = native.Flock(native.generate(5000, 1))
    straight = native.lib().flk_copies_straight
    w = f.read()[1]  # page-locked
    at = w.ctypes.data
    assert straight(at, w.nbytes) == straight(at + 60, w.nbytes - 60) == straight(at + w.nbytes - 4, 4) == 1
    assert [straight(at + k, 60) for k in (1, 2, 3)] == [0, 0, 0]
    assert straight(w.copy().ctypes.data, w.nbytes) == 0
    buf = np.zeros(8 * PAGE, dtype=np.uint8)
    p = buf.ctypes.data + (-buf.ctypes.data) % PAGE
    a, b = buf[p - buf.ctypes.data:][:PAGE], buf[p - buf.ctypes.data + 3 * PAGE:][:PAGE]
    with native.pinned(a, b):  # two pages page-locked, two between them not
        assert straight(p, PAGE) == straight(p + 3 * PAGE, PAGE) == straight(p + 4, PAGE - 4) == 1
        assert straight(p, 4 * PAGE) == 0  # both ends are
        assert straight(p, PAGE + 1) == straight(p + 4, PAGE) == straight(p + PAGE, 4) == 0
        assert straight(p - 4, PAGE) == 0
    assert straight(p, PAGE) == 0
    f.close()
