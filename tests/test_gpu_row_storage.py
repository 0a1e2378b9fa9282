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
