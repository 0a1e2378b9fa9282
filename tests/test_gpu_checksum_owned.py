"""The checksum of a list whose last build went to arrays of the caller is an
error, not that of an empty list."""

import pytest

from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_no_checksum_of_pairs_elsewhere(batch):
    import torch

    import vesin_b200
    from vesin_b200._sharded import list_checksum

    points, box, _ = W.diamond(3)
    points, box = torch.tensor(points, device="cuda"), torch.tensor(box, device="cuda")
    calculator = (vesin_b200.BatchNeighborList if batch else vesin_b200.NeighborList)(5.0, True)

    def build(copy):
        if batch:
            return calculator.compute(points, [0, len(points)], quantities="ijSd", copy=copy)[0]
        return calculator.compute(points, box, True, "ijSd", copy=copy)

    rows = len(build(copy=False)[0])
    checksum = list_checksum(calculator._neighbors)
    assert checksum[3] == rows > 0
    build(copy=True)
    with pytest.raises(RuntimeError, match="the list holds none"):
        list_checksum(calculator._neighbors)
    build(copy=False)
    assert list_checksum(calculator._neighbors) == checksum
