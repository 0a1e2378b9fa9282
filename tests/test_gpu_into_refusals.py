"""Arrays that vesin_b200_neighbors_into and vesin_b200_neighbors_batch_into
refuse before anything is written: not device memory, or not aligned to their
elements, whether the caller brings them or hands them out when asked."""

import ctypes

import numpy as np
import pytest

from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu

CAPACITY = 60000


@pytest.mark.parametrize("entry", ["single", "float", "sorted", "canonical", "skin", "batch"])
@pytest.mark.parametrize("when", ["brought", "allocated"])
def test_refused_arrays(entry, when):
    import torch

    from vesin_b200 import _c_api as api

    lib = api.get_library()
    device = torch.device("cuda", 0)
    points, box, periodic = W.diamond(3)
    dtype = torch.float32 if entry == "float" else torch.float64
    p, b = torch.tensor(points, device=device, dtype=dtype), torch.tensor(box, device=device, dtype=dtype)
    per = torch.tensor(periodic, device=device)
    value = dtype.itemsize
    room = torch.empty(CAPACITY * 24 + 64, dtype=torch.uint8, device=device)
    host = np.empty(CAPACITY * 24 + 64, dtype=np.uint8)
    good, on_host = room.data_ptr(), host.ctypes.data + (-host.ctypes.data) % 16
    options = api.VesinOptions()
    options.cutoff = 5.0
    options.full = True
    options.sorted = entry == "sorted"
    options.skin = 1.0 if entry == "skin" else 0.0
    flags = {"float": api.VESIN_B200_FLOAT32, "canonical": api.VESIN_B200_CANONICAL}.get(entry, 0)
    offsets = np.array([0, len(points)], dtype=np.uint64)
    pair_offsets = torch.empty(2, dtype=torch.int64, device=device)

    def build(**pointers):
        neighbors, length, error = api.VesinNeighborList(), ctypes.c_size_t(), ctypes.c_char_p()
        arrays = api.VesinB200Arrays()

        def fill(target):
            for name, pointer in pointers.items():
                setattr(target, name, pointer)
            target.capacity = CAPACITY
            return 0

        if when == "brought":
            fill(arrays)
        allocate = api.VesinB200Allocate(lambda _context, _n, target: fill(target.contents))
        tail = (ctypes.byref(neighbors), ctypes.byref(arrays), allocate, None)
        torch.cuda.synchronize()
        if entry == "batch":
            status = lib.vesin_b200_neighbors_batch_into(
                p.data_ptr(), offsets.ctypes.data, 1, None, None, api.VesinDevice(api.VesinCUDA, 0), options, flags, False, *tail,
                pair_offsets.data_ptr(), ctypes.byref(length), ctypes.byref(error),
            )
        else:
            status = lib.vesin_b200_neighbors_into(
                p.data_ptr(), len(points), b.data_ptr(), per.data_ptr(), api.VesinDevice(api.VesinCUDA, 0), options, flags, *tail,
                ctypes.byref(length), ctypes.byref(error),
            )
        lib.vesin_free(ctypes.byref(neighbors))
        return status, length.value, (error.value or b"").decode()

    needs = {"pairs": 16, "i": 8, "j": 8, "shifts": 4, "distances": value, "vectors": value}
    for name, alignment in needs.items():
        assert build(**{name: on_host}) == (1, 0, f"array `{name}` is not device memory on the CUDA device of `neighbors`")
        assert build(**{name: good + alignment // 2}) == (1, 0, f"array `{name}` is not aligned to {alignment} bytes")
        status, length, message = build(**{name: good})
        assert status == 0 and 0 < length <= CAPACITY, message
    # columns beside `pairs` are not written, nor looked at
    assert build(pairs=good, i=on_host)[0] == 0
