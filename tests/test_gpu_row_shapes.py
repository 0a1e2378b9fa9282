"""Sorted and canonical lists for every kind of CTA that decides and writes rows:
few units and many, that all fit a batch, a wide one, or neither; units that are
few because most of the box is empty. Compared with the unsorted list, whose
kernel is another one."""

import numpy as np
import pytest

import vesin_b200
from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _by_pair(values, n):
    import torch

    values = dict(zip("ijSdD", values))
    key = values["i"].view(torch.int64) * n + values["j"].view(torch.int64)
    order = torch.sort(key).indices
    return {name: value[order] for name, value in [("key", key), ("S", values["S"]), ("d", values["d"]), ("D", values["D"])]}


def _check(points, box, cutoff, full, canonical, dtype="float64", calculator=None):
    """(no pair of points has two images within the cutoff)"""
    import torch

    kind = getattr(torch, dtype)
    p, b = torch.tensor(points, device="cuda", dtype=kind), torch.tensor(box, device="cuda", dtype=kind)
    expected = _by_pair(vesin_b200.NeighborList(cutoff, full).compute(p, b, True, "ijSdD"), len(p))
    calculator = calculator or vesin_b200.NeighborList(cutoff, full, sorted=True, canonical=canonical)
    for _ in range(2):  # the second build knows how full the units are, and writes ahead
        values = calculator.compute(p, b, True, "ijSdD")
        i, j = values[0].view(torch.int64), values[1].view(torch.int64)
        assert bool((i[1:] >= i[:-1]).all())
        if canonical:
            assert bool(((i[1:] > i[:-1]) | (j[1:] > j[:-1])).all())
        got = _by_pair(values, len(p))
        for name in expected:
            assert torch.equal(got[name], expected[name]), name


@pytest.mark.parametrize("canonical", [False, True])
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize(
    "cells,cutoff",
    [
        (6, 5.0),  # 64 units of 330 candidates
        (16, 5.0),  # 1331
        (8, 7.0),  # 64 of 1728
        (18, 7.0),  # 729
        (10, 8.9),  # 64 of 3375
        (20, 7.9),  # 729 of 2370
    ],
)
def test_crystals(cells, cutoff, full, canonical, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, _ = W.diamond(cells, seed=cells)
    _check(points, box, cutoff, full, canonical, "float32" if cells == 16 else "float64")


@pytest.mark.parametrize("canonical", [False, True])
@pytest.mark.parametrize("n,cutoff", [(3000, 5.0), (8000, 7.0)])
def test_droplets(n, cutoff, canonical, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    rng = np.random.default_rng(n)
    radius = (3.0 * n / 0.1 / 4.0 / np.pi) ** (1.0 / 3.0)
    points = rng.normal(size=(n, 3))
    points *= (radius * rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(points, axis=1))[:, None]
    calculator = vesin_b200.NeighborList(cutoff, True, sorted=True, canonical=canonical)
    for scale in (1.0, 1.0, 1.01, 1.02, 0.9):  # (a new plan for every box)
        _check(points + 3.0 * radius, scale * 6.0 * radius * np.eye(3), cutoff, True, canonical, calculator=calculator)


@pytest.mark.parametrize("canonical", [False, True])
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n,cutoff", [(40, 9.0), (150, 11.0)])
def test_images_of_few_points(n, cutoff, full, canonical, monkeypatch):
    """Rows that go on from batch to batch and from group to group, with a shift for most pairs."""
    import torch

    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, periodic = W.small_triclinic(n, seed=n)
    calculator = vesin_b200.NeighborList(cutoff, full, sorted=True, canonical=canonical)
    expected = O.canonical(O.restated_neighbors(points, box, periodic, cutoff, full, "ijSdD"))
    for _ in range(2):
        got = {key: value.cpu().numpy() for key, value in zip("ijSdD", calculator.compute(torch.tensor(points, device="cuda"), torch.tensor(box, device="cuda"), True, "ijSdD"))}
        got["i"], got["j"] = got["i"].astype(np.int64), got["j"].astype(np.int64)
        assert np.all(np.diff(got["i"]) >= 0)
        if not canonical:
            got = O.canonical(got)
        for key in "ijSdD":
            assert np.array_equal(got[key], expected[key]), key


@pytest.mark.parametrize("span", [122879, 122880])
def test_span_of_indices_of_a_full_unit(span):
    """Units of about 1200 candidates, ranked by 8 warps: the indices around one corner lie exactly as far
    apart as has a bit each, or one further."""
    rng = np.random.default_rng(span)
    n, length, cutoff = 123500, 220.0, 15.6
    points = rng.uniform(0.0, length, (n, 3))
    from_corner = np.abs(points - length * np.round(points / length)).max(axis=1)
    around = np.argsort(from_corner)[: int((from_corner < 40.0).sum())]
    index = np.full(n, -1)
    index[around[:2]] = [0, span]
    index[around[2:]] = rng.choice(np.arange(1, span), len(around) - 2, replace=False)
    index[index < 0] = np.setdiff1d(np.arange(n), index[around])
    placed = np.empty_like(points)
    placed[index] = points
    _check(placed, length * np.eye(3), cutoff, True, True)
