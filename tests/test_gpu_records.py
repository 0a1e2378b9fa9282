"""Cell-sorted records: a point and its wrap shift in 32 bytes. Shifts beyond
the 10 bits a component has there ([-512, 511]) are kept beside the records;
the lists must not show the difference."""

import numpy as np
import pytest

from gpu_utils import gpu_compute
from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [200, 20000])  # one CTA sorts the small system, the chain of kernels the large one
@pytest.mark.parametrize("kind", [dict(full=True), dict(full=False), dict(full=True, sorted=True)])
def test_points_many_boxes_away(n, kind):
    points, box, periodic = W.liquid(n, seed=31)
    rng = np.random.default_rng(32)
    images = rng.choice([0, 0, -512, -513, 511, 512, 3000, -70000], (n, 3))
    points = points + images @ box
    got = O.canonical(gpu_compute(points, box, periodic, 5.0, **kind))
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 5.0, kind["full"], "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key
