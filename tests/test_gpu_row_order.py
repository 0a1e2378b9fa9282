"""Sorted and canonical lists around the sizes at which the row-writing kernel
changes its ways: all candidates of a unit in one batch of 1024 (of 896, in
the order of their indices, for canonical lists), in one of 2048, in several batches (the
rows are then sorted behind the kernel), and boxes with repeated indices."""

import numpy as np
import pytest

from gpu_utils import gpu_compute
from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _system(n, length, seed=3):
    rng = np.random.default_rng(seed)
    return rng.uniform(-0.3 * length, 0.7 * length, (n, 3)), length * np.eye(3), [True, True, True]


def _canonical_list(points, box, periodic, cutoff, full, dtype="float64"):
    import torch

    import vesin_b200

    calculator = vesin_b200.NeighborList(cutoff=cutoff, full_list=full, canonical=True)
    out = calculator.compute(
        torch.tensor(points, device="cuda", dtype=getattr(torch, dtype)), torch.tensor(box, device="cuda", dtype=getattr(torch, dtype)),
        periodic, "ijSdD",
    )
    return dict(zip("ijSdD", (t.cpu().numpy() for t in out)))


# 4 cells of the cutoff per direction: 27 / 64 of the points are candidates of a unit; the last
# box is shorter than two cutoffs, where an index comes more than once in a row
@pytest.mark.parametrize("n, length", [(33, 20.5), (1200, 20.5), (2100, 20.5), (2300, 20.5), (4700, 20.5), (5200, 20.5), (300, 9.0)])
@pytest.mark.parametrize("full", [True, False])
def test_canonical_order(n, length, full, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, periodic = _system(n, length)
    got = _canonical_list(points, box, periodic, 5.0, full)
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 5.0, full, "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key


@pytest.mark.parametrize("n, length", [(33, 20.5), (1200, 20.5), (2500, 20.5), (5200, 20.5), (300, 9.0)])
@pytest.mark.parametrize("full", [True, False])
def test_sorted_rows(n, length, full, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, periodic = _system(n, length, seed=4)
    got = gpu_compute(points, box, periodic, 5.0, full, sorted=True)
    assert np.all(np.diff(got["i"].astype(np.int64)) >= 0)
    got = O.canonical(got)
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 5.0, full, "ijSdD"))
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key


def test_canonical_order_float32_values():
    points, box, periodic = W.diamond(6, seed=2)
    points, box = points.astype(np.float32), box.astype(np.float32)
    got = _canonical_list(points, box, periodic, 5.0, True, dtype="float32")
    expected = O.canonical(O.restated_neighbors(points.astype(np.float64), box.astype(np.float64), periodic, 5.0, True, "ijSdD"))
    for key in "ijS":
        assert np.array_equal(got[key], expected[key]), key
    assert np.array_equal(got["d"], expected["d"].astype(np.float32)) and np.array_equal(got["D"], expected["D"].astype(np.float32))
