"""Launches of the general pair kernel with too many units to share any out, and
just few enough to: slabs, stencils of more than 64 cells, arrays that are not
aligned for paired stores."""

import numpy as np
import pytest

from gpu_utils import gpu_compute
from oracle import oracle as O
from test_gpu_into import test_arrays_of_the_caller as arrays_of_the_caller
from test_gpu_slab import _sharded_union
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _same(got, expected):
    got, expected = O.canonical(got), O.canonical(expected)
    for key in "ijSdD":
        assert np.array_equal(got[key], expected[key]), key


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n", [4000, 20000, 120000])
def test_slabs(n, full):
    points, box, periodic = W.liquid(n, seed=n)
    _same(_sharded_union(points, box, periodic, 6.0, full, 2), O.restated_neighbors(points, box, periodic, 6.0, full, "ijSdD"))


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n,length", [(12000, 380.0), (20000, 400.0)])
def test_thin_films(n, length, full):
    box, periodic = np.diag([length, length, 2.5]), [True, True, True]
    points = np.random.default_rng(n).uniform(0.0, 1.0, (n, 3)) @ box
    _same(gpu_compute(points, box, periodic, 6.0, full), O.restated_neighbors(points, box, periodic, 6.0, full, "ijSdD"))


@pytest.mark.parametrize("columns", [True, False])
@pytest.mark.parametrize("cells", [13, 14])
def test_unaligned_arrays(cells, columns, monkeypatch):
    crystal = W.diamond
    monkeypatch.setattr(W, "diamond", lambda _: crystal(cells))
    arrays_of_the_caller(full=True, columns=columns, offset=1)
