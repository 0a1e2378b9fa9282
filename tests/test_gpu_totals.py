"""The total that the last CTA of the pair kernel hands to the host is that of
all CTAs: counting passes and writing passes of one CTA, of fewer than there are
SMs and of more than are resident, over and over."""

import pytest

from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n", [1, 3, 9, 20])
def test_total_of_all_ctas(n, full):
    import torch

    import vesin_b200

    points, box, periodic = W.diamond(n)
    periodic = [False] * 3 if n == 1 else periodic
    expected = len(O.restated_neighbors(points, box, periodic, 3.0, full, "ij")["i"])
    points, box = torch.tensor(points, device="cuda"), torch.tensor(box, device="cuda")
    kept = vesin_b200.NeighborList(3.0, full)
    for _ in range(40):
        assert len(kept.compute(points, box, list(map(bool, periodic)), "ij")[0]) == expected
        # a new calculator counts first
        assert len(vesin_b200.NeighborList(3.0, full).compute(points, box, list(map(bool, periodic)), "ij")[0]) == expected
