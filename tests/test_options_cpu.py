"""The options that the calculators hand to the engine, without a GPU: those of
this call's quantities, in whatever container they come and whatever the last
call asked for."""

import numpy as np
import pytest

import vesin_b200

CALCULATORS = [vesin_b200.NeighborList, vesin_b200.BatchNeighborList, vesin_b200.ShardedNeighborList]


def _returned(options):
    return bool(options.return_shifts), bool(options.return_distances), bool(options.return_vectors)


@pytest.mark.parametrize("kind", CALCULATORS)
def test_a_list_that_changes_between_calls(kind):
    calculator = kind(cutoff=3.0, full_list=True)
    quantities = ["i", "j"]
    assert _returned(calculator._options(quantities)) == (False, False, False)
    quantities.append("D")
    assert _returned(calculator._options(quantities)) == (False, False, True)
    quantities[:] = ["S", "d"]
    assert _returned(calculator._options(quantities)) == (True, True, False)


@pytest.mark.parametrize("kind", CALCULATORS)
@pytest.mark.parametrize("container", [str, list, tuple, lambda letters: np.array(list(letters))])
def test_containers_of_letters(kind, container):
    def quantities(letters):
        return container(letters) if container is not str else letters

    calculator = kind(cutoff=3.0, full_list=True)
    for letters in ("ijd", "ijd", "ijS", "PSdD", "i"):
        assert _returned(calculator._options(quantities(letters))) == tuple(letter in letters for letter in "SdD")


def test_attributes_that_change_between_calls():
    calculator = vesin_b200.NeighborList(3.0, True)
    assert calculator._options("ij").cutoff == 3.0
    calculator.cutoff, calculator.full_list, calculator.skin, calculator.algorithm = 4.5, False, 0.5, "cell_list"
    options = calculator._options("ij")
    assert (options.cutoff, options.full, options.skin, options.algorithm) == (4.5, False, 0.5, 2)
