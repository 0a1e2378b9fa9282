"""The fp32 screen of the pair passes at the ends of the range of fp32: cutoffs
whose squares overflow, or nearly do, and clusters so far apart that the squares
of coordinates do. The exact predicate then decides every candidate."""

import numpy as np
import pytest

from gpu_utils import gpu_compute

pytestmark = pytest.mark.gpu


def _expected(points, cutoff):
    """Full list without periodicity, in the arithmetic of the predicate."""
    v = points[None] - points[:, None]
    d2 = (v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]) + v[..., 2] * v[..., 2]
    near = d2 < cutoff * cutoff
    np.fill_diagonal(near, False)
    return set(zip(*np.nonzero(near)))


@pytest.mark.parametrize("sorted", [False, True])
@pytest.mark.parametrize("cutoff", [1.0, 9.0e14, 1.1e15, 1.2e19, 1.5e19, 1.8e19, 1.0e20, 1.0e40])
@pytest.mark.parametrize("n", [65, 700])
def test_large_cutoffs(n, cutoff, sorted, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points = np.random.default_rng(3).random((n, 3)) * 4 * cutoff
    expected = _expected(points, cutoff)
    for full in (True, False):
        got = gpu_compute(points, np.zeros((3, 3)), [False] * 3, cutoff, full, "ij", sorted=sorted)
        pairs = set(zip(got["i"], got["j"]))
        assert len(pairs) == len(got["i"])
        assert pairs == (expected if full else {(i, j) for i, j in expected if i < j})


@pytest.mark.parametrize("sorted", [False, True])
def test_clusters_far_apart(sorted, monkeypatch):
    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    rng = np.random.default_rng(4)
    cutoff = 1.0e10
    centres = np.array([[0.0, 0.0, 0.0], [3.0e22, 0.0, 0.0], [1.0e22, 2.0e22, 3.0e22]])
    points = np.repeat(centres, 50, axis=0) + rng.uniform(-1.5, 1.5, (150, 3)) * cutoff
    got = gpu_compute(points, np.zeros((3, 3)), [False] * 3, cutoff, True, "ij", sorted=sorted)
    expected = _expected(points, cutoff)
    assert len(expected) > 500 and set(zip(got["i"], got["j"])) == expected
