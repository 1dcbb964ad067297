"""Where the host locks no pages everything still runs, on ordinary memory: the same
bits. (The failure is the host's: no GPU work differs.)"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def states(native, sizes):
    with native.Batch() as b:
        ids = [b.add(native.generate(n, n)) for n in sizes]
        b.step(3)
        b.step_each(ids[::2], [2 + k % 5 for k in range(len(ids[::2]))])
        b.step(12)
        return [b.read(i) for i in ids]


@pytest.mark.parametrize("sizes", [(500,), (20_000, 300), tuple(range(40, 90))])  # the last: a table that grows
def test_steps_and_results(native, sizes):
    want = states(native, sizes)
    try:
        native.lib().flk_debug_fail_locks(1 << 30)
        got = states(native, sizes)
    finally:
        native.lib().flk_debug_fail_locks(0)
    assert native.lib().flk_copies_straight(got[0][1].ctypes.data, got[0][1].nbytes) == 0
    assert all(t == u and x.tobytes() == y.tobytes() for (t, x), (u, y) in zip(got, want))
