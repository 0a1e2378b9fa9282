"""Canonical lists without shifts: distances and vectors come in the order of
the shifts all the same, where a box shorter than two cutoffs has a second index
several times in a row."""

import pytest

from test_gpu_row_order import _system
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["crystal", "short_box", "triclinic", "long_box"])
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("copy", [True, False])
def test_columns_of_the_whole_list(system, full, dtype, copy, monkeypatch):
    import torch

    import vesin_b200

    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, periodic = {"crystal": W.diamond(2), "short_box": _system(300, 9.0), "triclinic": W.small_triclinic(), "long_box": W.diamond(4)}[system]
    inputs = [torch.tensor(a, device="cuda", dtype=getattr(torch, dtype)) for a in (points, box)]
    periodic = torch.tensor(periodic, device="cuda")
    whole = dict(zip("ijSdD", vesin_b200.NeighborList(5.5, full, canonical=True).compute(*inputs, periodic, "ijSdD")))
    assert len(whole["i"]) > 0
    for quantities in ("ijd", "ijdD", "D"):
        columns = vesin_b200.NeighborList(5.5, full, canonical=True).compute(*inputs, periodic, quantities, copy=copy)
        for key, column in zip(quantities, columns):
            expected = whole[key]
            if key in "ij":
                column, expected = column.contiguous().view(torch.int64), expected.view(torch.int64)
            assert torch.equal(column, expected), (quantities, key)
