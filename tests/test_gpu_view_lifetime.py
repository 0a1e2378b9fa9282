"""Views of the library's arrays (copy=False) keep what they show alive: the
calculator may go out of scope before them."""

import gc

import numpy as np
import pytest

from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_views_outlive_the_calculator():
    import torch

    import vesin_b200

    points, box, periodic = W.diamond(3, seed=1)
    points, box = torch.tensor(points, device="cuda"), torch.tensor(box, device="cuda")

    def single():
        return vesin_b200.NeighborList(4.0, True).compute(points, box, periodic, "PSdD", copy=False)

    def batch():
        values, offsets = vesin_b200.BatchNeighborList(4.0, True).compute(points, [0, 100, len(points)], quantities="PSdD", copy=False)
        return (*values, offsets)

    for views_of in (single, batch):
        calculators = [o for o in gc.get_objects() if type(o) in (vesin_b200.NeighborList, vesin_b200.BatchNeighborList)]
        views = views_of()
        gc.collect()
        alive = [o for o in gc.get_objects() if type(o) in (vesin_b200.NeighborList, vesin_b200.BatchNeighborList)]
        assert len(alive) == len(calculators) + 1  # the views hold it (checked before any of their memory is read)
        assert np.all(views[2].cpu().numpy() < 4.0)
        del views, alive
        gc.collect()
        alive = [o for o in gc.get_objects() if type(o) in (vesin_b200.NeighborList, vesin_b200.BatchNeighborList)]
        assert len(alive) == len(calculators)
