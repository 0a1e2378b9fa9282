"""The histogram of the cells counts a warp's points cell by cell when
neighbours share one, and point by point when none do: the same lists for
points in lattice order, in random order and in orders between."""

import numpy as np
import pytest

from gpu_utils import gpu_compute
from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["lattice", "random", "runs", "one cell"])
def test_order_of_the_input(order):
    points, box, periodic = W.diamond(14, seed=3)  # 21 952 atoms: beyond the one-CTA front
    rng = np.random.default_rng(4)
    if order == "random":
        points = points[rng.permutation(len(points))]
    elif order == "runs":
        # random order with a pair of equal neighbours in some of the warps only
        points = points[rng.permutation(len(points))]
        points[1::64] = points[0::64] + 0.3
    elif order == "one cell":
        points = points[:20001]
        points[5000:5100] = points[5000] + rng.uniform(-0.2, 0.2, (100, 3))
    got = O.canonical(gpu_compute(points, box, periodic, 4.0, True))
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 4.0, True, "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key
