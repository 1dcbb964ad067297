"""Birds on both sides of the radius above which a whole warp decides them from the
outset (8.01 rows of 2.67 m / 4 = 5.34 m at the 4 m cell), against the oracle and
in a batch, whichever list and kernel takes them."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import assert_step_parity
from test_row_lattice import cube

pytestmark = pytest.mark.gpu

LINE = 5.34


@pytest.mark.parametrize("density", [0.5, 0.004])
@pytest.mark.parametrize("radius", [(LINE - 0.02, LINE + 0.02), (1.0, 9.0), (6.0, 8.0)])
def test_step_matches_the_oracle(native, oracle, density, radius):
    assert_step_parity(native, oracle, cube(8195, 50, radius=radius, density=density, due=0.4))


@pytest.mark.parametrize("cell", [2.5, 4.0, 6.0])
@pytest.mark.parametrize("staged", [0, 1])
def test_alone_and_in_a_batch(native, cell, staged):
    line = LINE * cell / 4.0
    flocks = [cube(n, 60 + n, radius=(0.8 * line, 1.2 * line), density=0.02, due=0.3) for n in (8192, 300, 12_001)]
    with native.Batch() as b:
        b.tune(cell=cell, staged=staged)
        ids = [b.add(w) for w in flocks]
        b.step(3)
        for i, w in zip(ids, flocks):
            with native.Flock(w) as f:
                f.tune_cell(cell)
                f.tune_decide(staged)
                f.step(3)
                assert f.read()[1].tobytes() == b.read(i)[1].tobytes()
