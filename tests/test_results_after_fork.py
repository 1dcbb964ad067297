"""A forked child has its own copy of the arrays that read() handed out: what the
parent reads into the same block later does not reach it, and what it writes
does not reach the parent."""
from __future__ import annotations

import os

import pytest

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore::DeprecationWarning")]


@pytest.mark.parametrize("n", [2000, 60_000])
def test_a_forked_child_keeps_its_array(native, n):
    f = native.Flock(native.generate(n, 2))
    f.step(2)
    w = f.read()[1]
    had = w.tobytes()
    at = w.ctypes.data
    to_child, go = os.pipe()
    pid = os.fork()
    if pid == 0:  # no GPU work, no return into pytest
        os.read(to_child, 1)
        same = w.tobytes() == had
        w[:] = -1.0
        os._exit(0 if same else 1)
    del w  # the block goes back, and one of the next results takes it
    f.step(2)
    results = [f.read()[1]]
    while results[-1].ctypes.data != at and len(results) < 100:
        results.append(f.read()[1])
    w = results[-1]
    want = w.tobytes()
    os.write(go, b"x")
    _, status = os.waitpid(pid, 0)
    os.close(go)
    os.close(to_child)
    assert w.ctypes.data == at and status == 0
    assert w.tobytes() == want == f.read()[1].tobytes()
    f.close()


def test_a_child_gives_no_block_back(native, monkeypatch):
    f = native.Flock(native.generate(2000, 2))
    w = f.read()[1]
    returned = []
    monkeypatch.setattr(native.lib(), "flk_host_free", returned.append, raising=False)
    pid = os.fork()
    if pid == 0:
        del w
        os._exit(len(returned))
    _, status = os.waitpid(pid, 0)
    assert status == 0 and not returned
    del w  # the parent's goes back
    assert len(returned) == 1
    monkeypatch.undo()
    native.lib().flk_host_free(returned[0])
    f.close()
