"""`periodic` beside numpy inputs: whatever numpy makes three flags of."""

import numpy as np
import pytest

from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "periodic",
    [
        [True, False, True], (1, 0, 1), [None, True, True], ["", "a", "b"], [np.array(True), True, False], np.array([2.5, 0.0, 1.0]), [object(), 0, 1.5],
    ],
    ids=str,
)
def test_flags_of_numpy(periodic):
    import vesin_b200

    points, box, _ = W.diamond(3)
    calculator = vesin_b200.NeighborList(5.0, True)
    flags = [bool(flag) for flag in periodic]
    expected = calculator.compute(points, box, np.array(flags), "ij")
    got = calculator.compute(points, box, periodic, "ij")
    assert len(got[0]) == len(expected[0]) and np.array_equal(np.bincount(got[0].astype(np.int64)), np.bincount(expected[0].astype(np.int64)))


@pytest.mark.parametrize("periodic", [[True, True], [[True], [True], [True]], np.array(True)], ids=str)
def test_refused_flags(periodic):
    import vesin_b200

    points, box, _ = W.diamond(3)
    with pytest.raises(ValueError, match="`periodic` must be a single boolean or a sequence of three booleans"):
        vesin_b200.NeighborList(5.0, True).compute(points, box, periodic, "ij")
