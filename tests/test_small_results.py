"""Results on both sides of the size (128 KiB) up to which ordinary memory gets them
by way of the engine's page-locked block. Bit-exact: the words are moved."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 136, 137, 2184, 2185])
@pytest.mark.parametrize("off", [0, 1, 60])
def test_every_word_and_nothing_beside_it(native, n, off):
    words = native.generate(n, n)
    raw = np.full(n * 60 + 256, 0x5A, dtype=np.uint8)
    out = np.frombuffer(raw, "<f4", n * 15, offset=64 + off).reshape(n, 15)
    with native.Flock(words) as f, native.Batch() as b:
        i = b.add(words)
        assert f.read(out)[1].tobytes() == words.tobytes() == b.read(i)[1].tobytes()
        f.step(5)
        b.step(5)
        assert f.read(out)[1].tobytes() == b.read(i)[1].tobytes() != words.tobytes()
        assert (raw[:64 + off] == 0x5A).all() and (raw[64 + off + n * 60:] == 0x5A).all()
        native.lib().flk_debug_fail_locks(1 << 30)
        try:  # without the block
            assert native.Flock(words).read(out)[1].tobytes() == words.tobytes()
        finally:
            native.lib().flk_debug_fail_locks(0)
