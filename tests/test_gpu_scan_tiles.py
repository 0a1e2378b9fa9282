"""Scans of one launch (up to four tiles of 2048 elements) and of two, around
the line between them: cells of an unsorted list, rows of a sorted one."""

import numpy as np
import pytest

from gpu_utils import gpu_compute
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(n, cells, **kind):
    rng = np.random.default_rng(n)
    length = cells + 0.001
    points, box, periodic = rng.uniform(0.0, length, (n, 3)), length * np.eye(3), [True, True, True]
    got = O.canonical(gpu_compute(points, box, periodic, 1.0, True, **kind))
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 1.0, True, "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key


@pytest.mark.parametrize("cells", [12, 13, 20, 21])  # 1728, 2197, 8000 and 9261 cells
def test_cells(cells):
    _check(20000, cells)


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 8192, 8193])
def test_rows(n):
    _check(n, 12, sorted=True)
