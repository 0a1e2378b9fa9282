"""Sorted lists whose hit words need more storage than a uniform density would:
the deciding pass runs out of it, the host grows it and decides again."""

import numpy as np
import pytest

import vesin_b200
from gpu_utils import gpu_compute
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("canonical", [False, True])
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n,radius", [(700, 4.0), (2600, 7.0)])
def test_dense_cluster_in_a_large_box(n, radius, full, canonical, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    rng = np.random.default_rng(n)
    points = np.concatenate([rng.uniform(0.0, radius, (n, 3)), rng.uniform(0.0, 60.0, (n // 10, 3))])
    points = points[rng.permutation(len(points))]
    box, periodic = 60.0 * np.eye(3), [True, True, True]
    calculator = vesin_b200.NeighborList(3.0, full, sorted=True, canonical=canonical)
    expected = O.canonical(O.restated_neighbors(points, box, periodic, 3.0, full, "ijSdD"))
    for _ in range(2):
        values = dict(zip("ijSdD", calculator.compute(points, box, periodic, "ijSdD")))
        values["i"], values["j"] = values["i"].astype(np.int64), values["j"].astype(np.int64)
        assert np.all(np.diff(values["i"]) >= 0)
        if not canonical:
            values = O.canonical(values)
        for key in "ijSdD":
            assert np.array_equal(values[key], expected[key]), key


@pytest.mark.parametrize("copy", [False, True])
@pytest.mark.parametrize("canonical", [False, True])
@pytest.mark.parametrize("full", [True, False])
def test_rows_written_ahead(full, canonical, copy, monkeypatch):
    """The rows of a list that was built before are written before the host has seen how many there
    are: into arrays that hold them, that are too short, for units with more candidates than the
    last build had, and behind a plan that is refused."""
    import torch

    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    rng = np.random.default_rng(5)
    n, length = 3000, 24.0
    loose = rng.uniform(0.0, length, (n, 3))
    dense = np.where(rng.random((n, 1)) < 0.6, rng.uniform(0.0, 6.0, (n, 3)), loose)
    denser = np.where(rng.random((n, 1)) < 0.9, rng.uniform(0.0, 5.0, (n, 3)), loose)
    box, periodic = length * np.eye(3), [True, True, True]
    moved = loose + rng.uniform(-0.1, 0.1, loose.shape)
    calculator = vesin_b200.NeighborList(3.0, full, sorted=True, canonical=canonical)
    steps = [(loose, box), (moved, box), (dense, box), (denser, box), (denser, box), (moved, box), (moved, 1.2 * box), (moved[:1700], box), (loose, box)]
    for points, cell in steps:
        values = calculator.compute(torch.tensor(points, device="cuda"), torch.tensor(cell, device="cuda"), periodic, "ijSdD", copy=copy)
        values = {key: value.cpu().numpy() for key, value in zip("ijSdD", values)}
        values["i"], values["j"] = values["i"].astype(np.int64), values["j"].astype(np.int64)
        expected = O.canonical(O.restated_neighbors(points, cell, periodic, 3.0, full, "ijSdD"))
        assert np.all(np.diff(values["i"]) >= 0)
        if not canonical:
            values = O.canonical(values)
        for key in "ijSdD":
            assert np.array_equal(values[key], expected[key]), key
