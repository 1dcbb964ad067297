"""flk_grid_noalloc by separate launches (what runs where a device cannot hold the
one kernel's blocks together), and after calls whose barrier counters were left
in any state. Integers throughout: exact."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import DeviceBuffers

pytestmark = pytest.mark.gpu


class Grid:
    """One flock's call, its buffers kept."""

    def __init__(self, native, oracle, bufs, n):
        words = native.generate(n, n)
        self.n, self.B, self.lib, self.bufs = n, native.buckets_for(n), native.lib(), bufs
        self.want = oracle.grid(words, self.B)
        pos4 = np.zeros((n, 4), dtype=np.float32)
        pos4[:, :3] = words[:, :3]
        self.at = [bufs.upload(pos4), bufs.alloc(n * 4), bufs.alloc((self.B + 1) * 4), bufs.alloc(n * 4)]

    def check(self, separate=0, spoil=0):
        p, k, o, s = (C.c_void_p(x) for x in self.at)
        rc = self.lib.flk_debug_grid_noalloc(p, C.c_uint32(self.n), k, o, s, None, separate, spoil)
        assert rc == 0, self.lib.flk_last_error()
        got = [self.bufs.download(x, c) for x, c in zip(self.at[1:], (self.n, self.B + 1, self.n))]
        assert all(np.array_equal(g, w) for g, w in zip(got, self.want))


@pytest.mark.parametrize("n", [1, 33, 1023, 1025, 16_385, 32_769, 131_072])
def test_separate_launches(native, oracle, n):
    bufs = DeviceBuffers()
    try:
        g = Grid(native, oracle, bufs, n)
        for separate in (1, 0, 1):
            g.check(separate)
    finally:
        bufs.free()


def test_calls_after_spoilt_counters(native, oracle):
    bufs = DeviceBuffers()
    try:
        small, large = Grid(native, oracle, bufs, 3000), Grid(native, oracle, bufs, 100_000)
        for k in range(70):  # every set of counters more than twice
            (small, large)[k % 2].check(separate=k % 7 == 3, spoil=k % 3 != 2)
    finally:
        bufs.free()
