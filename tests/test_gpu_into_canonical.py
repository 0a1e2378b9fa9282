"""Canonical lists written into arrays of the caller that have the alignment of
their elements and no more (vesin_b200_neighbors_into): rows that come out of
the writing pass in their final order, and rows that are sorted behind it (a box
shorter than two cutoffs; more candidates per unit than a CTA orders)."""

import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_row_order import _system
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["in_order", "short_box", "many_candidates"])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("columns", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_canonical_arrays_of_the_caller(system, dtype, columns, offset, monkeypatch):
    import torch

    from vesin_b200 import _c_api as api

    monkeypatch.setenv("VESIN_CUDA_MAX_PAIRS_PER_POINT", "100000")
    points, box, periodic = {"in_order": W.diamond(5), "short_box": _system(300, 9.0), "many_candidates": _system(5200, 20.5)}[system]
    points, box = points.astype(dtype), box.astype(dtype)
    expected = O.canonical(O.restated_neighbors(points.astype(np.float64), box.astype(np.float64), periodic, 5.0, True, "ijSdD"))
    n = len(expected["i"])

    lib = api.get_library()
    device = torch.device("cuda", 0)
    p, b = torch.tensor(points, device=device), torch.tensor(box, device=device)
    per = torch.tensor(np.asarray(periodic), device=device)
    value = getattr(torch, dtype)
    size = 4 if dtype == "float32" else 8
    ij = torch.full((2 * (n + offset + 1),), -1, dtype=torch.int64, device=device)
    # (one component off the alignment of the allocation)
    S = torch.full((3 * n + offset,), -99, dtype=torch.int32, device=device)
    d = torch.full((n + offset,), -1.0, dtype=value, device=device)
    D = torch.full((3 * n + offset,), -1.0, dtype=value, device=device)
    arrays = api.VesinB200Arrays()
    if columns:
        arrays.i, arrays.j = ij.data_ptr() + 8 * offset, ij.data_ptr() + 8 * (n + 1 + offset)
    else:
        arrays.pairs = ij.data_ptr() + 16 * offset
    arrays.shifts, arrays.distances, arrays.vectors = S.data_ptr() + 4 * offset, d.data_ptr() + size * offset, D.data_ptr() + size * offset
    arrays.capacity = n

    options = api.VesinOptions()
    options.cutoff = 5.0
    options.full = True
    neighbors, length, error = api.VesinNeighborList(), ctypes.c_size_t(), ctypes.c_char_p()
    flags = api.VESIN_B200_CANONICAL | (api.VESIN_B200_FLOAT32 if dtype == "float32" else 0)
    torch.cuda.synchronize()
    status = lib.vesin_b200_neighbors_into(
        p.data_ptr(), len(points), b.data_ptr(), per.data_ptr(), api.VesinDevice(api.VesinCUDA, 0), options, flags, ctypes.byref(neighbors),
        ctypes.byref(arrays), api.VesinB200Allocate(lambda *_: 1), None, ctypes.byref(length), ctypes.byref(error),
    )
    assert status == 0 and length.value == n, error.value
    lib.vesin_free(ctypes.byref(neighbors))

    ij = ij.cpu().numpy()
    i, j = (ij[offset : offset + n], ij[n + 1 + offset : 2 * n + 1 + offset]) if columns else ij[2 * offset : 2 * offset + 2 * n].reshape(-1, 2).T
    assert np.array_equal(i, expected["i"]) and np.array_equal(j, expected["j"])
    assert np.array_equal(S[offset:].cpu().numpy().reshape(-1, 3), expected["S"])
    assert np.array_equal(d[offset:].cpu().numpy(), expected["d"].astype(dtype))
    assert np.array_equal(D[offset:].cpu().numpy().reshape(-1, 3), expected["D"].astype(dtype))
