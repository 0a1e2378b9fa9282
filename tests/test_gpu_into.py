"""Lists written straight into arrays of the caller
(vesin_b200_neighbors_into, vesin_b200_neighbors_batch_into): the same pairs as
in the library's own arrays, bit for bit, with the indices as (i, j) pairs or
as two columns, aligned for the paired stores or not, and whatever number of
pairs the arrays were sized for."""

import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _numpy(outputs, quantities="ijSdD"):
    result = {key: value.cpu().numpy() for key, value in zip(quantities, outputs)}
    for key in "ij":
        result[key] = result[key].astype(np.int64)
    return O.canonical(result)


def _same(a, b):
    for key in "ijSdD":
        assert np.array_equal(a[key], b[key]), key


@pytest.mark.parametrize("order", ["any", "sorted", "canonical"])
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_own_tensors_hold_what_views_hold(order, full, dtype):
    import torch

    import vesin_b200

    device = torch.device("cuda", 0)
    kind = dict(sorted=order == "sorted", canonical=order == "canonical")
    calculator = vesin_b200.NeighborList(5.0, full, **kind)
    # growing, shrinking and empty lists through one calculator
    for points, box, periodic in (W.diamond(3), W.diamond(9), W.cluster(), W.diamond(6), (np.zeros((1, 3)), np.zeros((3, 3)), np.array([False] * 3))):
        inputs = [torch.tensor(points, device=device).to(getattr(torch, dtype)), torch.tensor(box, device=device).to(getattr(torch, dtype))]
        own = calculator.compute(*inputs, periodic.tolist(), "ijSdD")
        viewed = vesin_b200.NeighborList(5.0, full, **kind)  # (its arrays go with it)
        views = viewed.compute(*inputs, periodic.tolist(), "ijSdD", copy=False)
        assert all(a.dtype == b.dtype and a.shape == b.shape and a.is_contiguous() for a, b in zip(own, views))
        if order != "any":
            assert torch.equal(own[0].view(torch.int64), views[0].contiguous().view(torch.int64))
        _same(_numpy(own), _numpy(views))
        pairs, i = calculator.compute(*inputs, periodic.tolist(), "Pi")
        assert pairs.shape == (len(i), 2)


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("columns", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_arrays_of_the_caller(full, columns, offset):
    """`offset` moves every array one element off the alignment that paired
    stores need (pairs stay on their 16 bytes)."""
    import torch

    from vesin_b200 import _c_api as api

    lib = api.get_library()
    device = torch.device("cuda", 0)
    points, box, periodic = W.diamond(5)
    p, b, per = torch.tensor(points, device=device), torch.tensor(box, device=device), torch.tensor(periodic, device=device)
    options = api.VesinOptions()
    options.cutoff = 5.0
    options.full = full
    neighbors = api.VesinNeighborList()
    arrays = api.VesinB200Arrays()
    length = ctypes.c_size_t()
    error = ctypes.c_char_p()
    held = {}

    @api.VesinB200Allocate
    def allocate(_context, n, target):
        held.clear()
        target = target.contents
        held["ij"] = torch.full((2 * (n + offset + 1),), -1, dtype=torch.int64, device=device)
        held["S"] = torch.empty((n + offset, 3), dtype=torch.int32, device=device)
        held["d"] = torch.empty(n + offset, dtype=torch.float64, device=device)
        held["D"] = torch.empty((n + offset, 3), dtype=torch.float64, device=device)
        base = held["ij"].data_ptr()
        if columns:
            target.i, target.j = base + 8 * offset, base + 8 * (n + 1 + 2 * offset)
        else:
            target.pairs = base + 16 * offset
        target.shifts, target.distances, target.vectors = (held[k].data_ptr() + size * offset for k, size in (("S", 12), ("d", 8), ("D", 24)))
        target.capacity = n
        return 0

    for _ in range(2):  # the second build has the arrays it needs
        status = lib.vesin_b200_neighbors_into(
            p.data_ptr(), len(points), b.data_ptr(), per.data_ptr(), api.VesinDevice(api.VesinCUDA, 0), options, 0, ctypes.byref(neighbors),
            ctypes.byref(arrays), allocate, None, ctypes.byref(length), ctypes.byref(error),
        )
        assert status == 0, error.value
        n = length.value
        assert neighbors.length == 0 and arrays.capacity == n
        ij = held["ij"].cpu().numpy()
        if columns:
            i, j = ij[offset : offset + n], ij[n + 1 + 2 * offset : 2 * n + 1 + 2 * offset]
        else:
            i, j = ij[2 * offset : 2 * offset + 2 * n].reshape(-1, 2).T
        got = {"i": i, "j": j, **{k: held[k][offset:].cpu().numpy() for k in "SdD"}}
        _same(O.canonical(got), O.canonical(O.restated_neighbors(points, box, periodic, 5.0, full, "ijSdD")))
    lib.vesin_free(ctypes.byref(neighbors))


def test_failed_allocation_is_an_error():
    import torch

    from vesin_b200 import _c_api as api

    lib = api.get_library()
    device = torch.device("cuda", 0)
    points, box, periodic = W.diamond(3)
    p, b, per = torch.tensor(points, device=device), torch.tensor(box, device=device), torch.tensor(periodic, device=device)
    options = api.VesinOptions()
    options.cutoff = 5.0
    neighbors, arrays, length, error = api.VesinNeighborList(), api.VesinB200Arrays(), ctypes.c_size_t(), ctypes.c_char_p()
    refuse = api.VesinB200Allocate(lambda _context, _n, _arrays: 1)
    status = lib.vesin_b200_neighbors_into(
        p.data_ptr(), len(points), b.data_ptr(), per.data_ptr(), api.VesinDevice(api.VesinCUDA, 0), options, 0, ctypes.byref(neighbors),
        ctypes.byref(arrays), refuse, None, ctypes.byref(length), ctypes.byref(error),
    )
    assert status == 1 and error.value == b"failed to allocate memory" and length.value == 0
    lib.vesin_free(ctypes.byref(neighbors))


@pytest.mark.parametrize("full", [True, False])
def test_batches(full):
    import torch

    import vesin_b200

    device = torch.device("cuda", 0)
    points, offsets = W.molecule_batch(n_systems=50, seed=8)
    points = torch.tensor(points, device=device)
    calculator = vesin_b200.BatchNeighborList(4.0, full)
    for last in (3, 50, 1, 50):
        inputs = (points[: offsets[last]], offsets[: last + 1])
        own, own_offsets = calculator.compute(*inputs, quantities="ijSdD", global_indices=True)
        viewed = vesin_b200.BatchNeighborList(4.0, full)
        views, view_offsets = viewed.compute(*inputs, quantities="ijSdD", global_indices=True, copy=False)
        assert torch.equal(own_offsets, view_offsets) and calculator.n_pairs == len(own[0])
        _same(_numpy(own), _numpy(views))
