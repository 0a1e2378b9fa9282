"""Launches of few units (64 candidates per batch, shared out to many CTAs) on
both sides of the line where ordinary batches take over."""

import numpy as np
import pytest

from gpu_utils import gpu_compute
from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("cells", [1, 2, 3, 5, 6, 7, 8])
def test_small_crystals(cells, full):
    points, box, periodic = W.diamond(cells, seed=cells)
    got = O.canonical(gpu_compute(points, box, periodic, 5.0, full))
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 5.0, full, "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n", [1, 33, 65, 150])
def test_cells_full_of_images(n, full, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, periodic = W.small_triclinic(n, seed=n)
    got = O.canonical(gpu_compute(points, box, periodic, 9.0, full))
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 9.0, full, "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key
