"""Quantities in a list that the caller changes between two calls, or in an
array of letters: every call returns what it is asked for."""

import numpy as np
import pytest

import vesin_b200
from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu

STEPS = ("ij", "ijD", "ijdD", "ijSdD", "ijS")


def _check(values, letters, points, box, periodic):
    values = {key: np.asarray(value.cpu() if hasattr(value, "cpu") else value) for key, value in zip(letters, values)}
    expected = O.restated_neighbors(points, box, periodic, 3.0, True, "ijSdD")
    # (pairs come in any order: columns are compared sorted)
    assert len(values["i"]) == len(expected["i"])
    for key in letters:
        assert np.allclose(np.sort(values[key].astype(float), axis=0), np.sort(expected[key].astype(float), axis=0), rtol=1e-12, atol=0.0), key


@pytest.mark.parametrize("container", [list, np.array])
@pytest.mark.parametrize("copy", [True, False])
@pytest.mark.parametrize("host", [True, False])
def test_quantities_that_change_between_calls(container, copy, host):
    import torch

    points, box, periodic = W.diamond(4, seed=2)
    inputs = (points, box) if host else (torch.tensor(points, device="cuda"), torch.tensor(box, device="cuda"))
    calculator = vesin_b200.NeighborList(3.0, True)
    kept = []
    for letters in STEPS:
        kept[:] = letters
        _check(calculator.compute(*inputs, True, kept if container is list else np.array(kept), copy=copy), letters, points, box, periodic)


@pytest.mark.parametrize("container", [list, np.array])
@pytest.mark.parametrize("copy", [True, False])
def test_quantities_of_batches_that_change_between_calls(container, copy):
    import torch

    points, box, periodic = W.diamond(4, seed=2)
    inputs = [torch.tensor(a, device="cuda")[None] for a in (box, periodic)]
    calculator = vesin_b200.BatchNeighborList(3.0, True)
    kept = []
    for letters in STEPS:
        kept[:] = letters
        values, _ = calculator.compute(
            torch.tensor(points, device="cuda"), np.array([0, len(points)]), *inputs, kept if container is list else np.array(kept), copy=copy
        )
        _check(values, letters, points, box, periodic)
