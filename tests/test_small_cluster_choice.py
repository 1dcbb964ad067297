"""Which batches run as one cluster per flock, of how many thread blocks, and that
each cluster size runs and gives the separate kernels' bits. How many clusters of
each size fit on the GPU at once is the device's own (seven to nine of 16 blocks on
the GB300s seen), so the counts on both sides of each line are taken from it. And
the autotuner's knobs where the launch shapes have no effect."""
from __future__ import annotations

import pytest

from test_autotune import FakeBatch, _autotune
from test_small_clusters import states

SIZES = (16, 8, 4, 2, 1)  # thread blocks per cluster
LARGEST = {c: min(4096, 512 * c) for c in SIZES}  # birds a cluster of each size takes


@pytest.fixture(scope="module")
def fit(native):
    """The most flocks that run as clusters of each size."""
    most = {}
    with native.Batch() as b:
        assert b.small_ctas() == 0
        for k in range(1, 400):
            b.add(native.generate(1, k))
            c = b.small_ctas()
            if not c:
                break
            most[c] = k
    return most


@pytest.mark.gpu
def test_every_cluster_size_is_in_use(fit):
    assert tuple(fit) == SIZES and list(fit.values()) == sorted(set(fit.values()))


@pytest.mark.gpu
@pytest.mark.parametrize("ctas", SIZES)
@pytest.mark.parametrize("more, above", [(0, 0), (0, 1), (1, 0), (1, -1)])
def test_choice_and_results(native, fit, ctas, more, above):
    flocks, largest = fit[ctas] + more, LARGEST[ctas] + above
    want = next((c for c in SIZES if flocks <= fit[c] and largest <= LARGEST[c]), 0)
    sizes = [1 + (7 * k * k) % 97 for k in range(flocks)]
    sizes[0] = sizes[flocks // 2] = sizes[-1] = largest
    with native.Batch() as b:
        for k, n in enumerate(sizes):
            b.add(native.generate(n, 1 + k))
        assert b.small_ctas() == want
        b.step(30)  # one kernel needs no graph; the separate ones capture the step graph
        assert b.graph_counts()[0] == (0 if want else 1)
    if want:
        for (t, x), (u, y) in zip(states(sizes), states(sizes, extra=(4097,))):
            assert t == u and x.tobytes() == y.tobytes()


def test_the_tuner_tries_only_the_cell_where_clusters_run(tmp_path, monkeypatch):
    at = _autotune()
    monkeypatch.setattr(at, "CACHE", str(tmp_path / "autotune.json"))
    b = FakeBatch(lambda s: 1.0 + 0.1 * (s["cell"] != 3.5) - 0.1 * (s["stream_bps"] == 16))  # the second is noise
    b.small_ctas = lambda: 8
    r = at.tune(b, steps=10, use_cache=False)
    assert r["shape"] == dict(at.DEFAULT, cell=3.5) and r["trials"] == len(at.SPACE["cell"])
