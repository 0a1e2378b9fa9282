"""Batches of periodic systems: tiles of 32 home points, chunks of 128 points
and batches of 256 images, at and around their edges; cells much smaller and
much larger than the cutoff; points many cells away from each other."""

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_batch import _check_batch

pytestmark = pytest.mark.gpu


def _cells(sizes, density, seed, thin=None):
    rng = np.random.default_rng(seed)
    points, boxes = [], []
    for n in sizes:
        box = np.diag(rng.uniform(1.0, 1.4, 3))
        box[1, 0], box[2, 0], box[2, 1] = rng.uniform(-0.6, 0.6, 3)
        if thin is not None:
            box[thin] *= 0.15
        box *= (max(n, 1) / density / abs(np.linalg.det(box))) ** (1.0 / 3.0)
        points.append(rng.uniform(0.0, 1.0, (n, 3)) @ box)
        boxes.append(box)
    return points, np.array(boxes)


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("flags", [(True, True, True), (True, False, True), (False, True, False), (False, False, False)])
def test_sizes_around_tiles_and_chunks(full, flags, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    sizes = [1, 2, 0, 31, 32, 33, 97, 127, 128, 129, 161, 256, 300]
    systems, boxes = _cells(sizes, 0.1, seed=5)
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    _check_batch(np.concatenate(systems), offsets, boxes, np.array([flags] * len(sizes)), 4.3, full, global_indices=True)


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("thin", [0, 2])
def test_thin_cells_and_far_points(full, thin, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    sizes = [1, 3, 40, 130]
    systems, boxes = _cells(sizes, 0.1, seed=6, thin=thin)
    rng = np.random.default_rng(7)
    # cells apart, then so far apart that the products with the shift round
    for reach in (4, 150000):
        moved = [p + rng.integers(-reach, reach + 1, (len(p), 3)) @ b for p, b in zip(systems, boxes)]
        offsets = np.concatenate([[0], np.cumsum(sizes)])
        _check_batch(np.concatenate(moved), offsets, boxes, np.ones((4, 3), dtype=bool), 6.0, full)


def test_many_systems_share_no_cta():
    """More systems than the GPU has CTAs for: one CTA per system walks all of its tiles."""
    import torch

    import vesin_b200

    sizes = [40] * 4000
    systems, boxes = _cells(sizes[:20], 0.1, seed=8)
    points = np.concatenate(systems * 200)
    offsets = np.arange(4001) * 40
    (i, j), pair_offsets = vesin_b200.BatchNeighborList(4.0, True).compute(
        torch.tensor(points, device="cuda"), offsets, torch.tensor(np.concatenate([boxes] * 200), device="cuda"),
        torch.ones((4000, 3), dtype=torch.bool, device="cuda"), "ij",
    )
    expected = [len(O.restated_neighbors(p, b, [True] * 3, 4.0, True, "ij")["i"]) for p, b in zip(systems, boxes)]
    assert np.array_equal(np.diff(pair_offsets.cpu().numpy()), np.array(expected * 200))
