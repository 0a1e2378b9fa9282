"""The filter of cached candidates reads the rows that the kernel in front of it
writes, and is launched while that one still runs: distances of the points as
they are now, call after call, for systems of one CTA up to many."""

import numpy as np
import pytest

from test_gpu_verlet import _same_as_oracle, _step
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 700, 9000])
def test_rows_of_this_call(n):
    import vesin_b200

    points, box, periodic = W.liquid(n, seed=11)
    rng = np.random.default_rng(3)
    cutoff = min(4.0, 0.45 * box[0, 0])
    calculator = vesin_b200.NeighborList(cutoff=cutoff, full_list=False, skin=1.0)
    for step in range(8):
        # everyone somewhere else, nobody further than half the skin from where the candidates were found
        moved = points + rng.uniform(-0.25, 0.25, points.shape)
        _same_as_oracle(_step(calculator, moved, box, periodic), moved, box, periodic, cutoff, False, label=f"step {step}")
