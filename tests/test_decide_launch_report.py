"""decide_occupancy reports the launch that the flock's steps use: the engine's own
choice by the flock's size (768, 896 or 1,024 threads per CTA and SM), and the
configured 1,024 once memory is reserved or another decide kernel is set."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, threads", [(9000, 768), (100_000, 768), (1_000_000, 896), (12_000_000, 1024)])
def test_threads_follow_the_flock(native, n, threads):
    with native.Flock(native.generate(n, 1)) as f:
        occ = f.decide_occupancy()
        own = occ["smem_bytes"] // (threads // 32)
        assert occ["threads"] == threads and occ["blocks_per_sm"] == 1
        assert own * (threads // 32) == occ["smem_bytes"]
        occ = f.decide_occupancy(1000)
        assert occ["threads"] == 1024 and occ["smem_bytes"] == own * 32 + 1000
        assert f.decide_occupancy()["threads"] == threads
        f.tune_decide(1)
        assert f.decide_occupancy()["threads"] == 1024
