"""Output tensors of the calculators: lists that the caller owns are written by
the engine straight into tensors of torch's allocator (``vesin_b200_neighbors_into``),
instead of being copied out of the library's arrays. A copy moves every byte of
the list twice more, and an index column picked out of the (i, j) pairs moves
twice as much again: at 45.6 M pairs that took 0.98 ms beside a build of 0.61 ms."""

import threading

import torch

from ._c_api import VesinB200Allocate, VesinB200Arrays

_active = threading.local()


# the address of the current stream without the object that torch wraps it in (a few us)
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def wait_for_caller(device):
    """The engine works on a stream of its own, which only the legacy default
    stream is ordered with: on any other stream, what the caller has queued
    (inputs being made, memory that a stream-ordered allocator has handed out)
    must be done before the engine touches it."""
    if _raw_stream is not None and device.index is not None and _raw_stream(device.index) == 0:
        return
    stream = torch.cuda.current_stream(device)
    if stream.cuda_stream != 0:
        stream.synchronize()


@VesinB200Allocate
def allocate_callback(_context, n_pairs, arrays):
    """Called by the engine, on the thread that called it, when a list needs
    more room than the arrays it was given have."""
    try:
        _active.outputs.allocate(n_pairs)
        wait_for_caller(_active.outputs.device)
        return 0
    except BaseException as error:  # nothing may propagate through the engine: the caller raises it
        _active.outputs.error = error
        return 1


class OutputTensors:
    """The tensors of one list: one per quantity asked for. Use as a context
    manager around the call that fills them."""

    def __init__(self, quantities, device, index_dtype, value_dtype):
        self.quantities = quantities
        self.device = device
        self.index_dtype = index_dtype
        self.value_dtype = value_dtype
        self.arrays = VesinB200Arrays()
        self.i = self.j = self.pairs = self.shifts = self.distances = self.vectors = None
        self.error = None

    def __enter__(self):
        self._outer = getattr(_active, "outputs", None)
        _active.outputs = self
        return self

    def __exit__(self, *_):
        _active.outputs = self._outer

    def allocate_guess(self, last, n_points):
        """Room for as many pairs per point as the last list had (`last`: its
        pairs and points), so that the engine can write at once. Where there is
        no such room the engine counts first and asks for what the list needs."""
        last_pairs, last_points = last
        if last_pairs == 0:
            return
        expected = last_pairs if n_points == last_points else last_pairs * n_points // last_points
        try:
            self.allocate(expected + expected // 16 + 64)
        except torch.cuda.OutOfMemoryError:
            self.release()

    def release(self):
        self.i = self.j = self.pairs = self.shifts = self.distances = self.vectors = None
        arrays = self.arrays
        arrays.capacity = 0
        arrays.i = arrays.j = arrays.pairs = arrays.shifts = arrays.distances = arrays.vectors = None

    def allocate(self, n_pairs):
        quantities, device, arrays = self.quantities, self.device, self.arrays
        if arrays.capacity != 0:
            self.release()  # what there is too little of goes back to the allocator first
        if "P" in quantities:
            self.pairs = torch.empty((n_pairs, 2), dtype=self.index_dtype, device=device)
            arrays.pairs = self.pairs.data_ptr()
        else:
            if "i" in quantities:
                self.i = torch.empty(n_pairs, dtype=self.index_dtype, device=device)
                arrays.i = self.i.data_ptr()
            if "j" in quantities:
                self.j = torch.empty(n_pairs, dtype=self.index_dtype, device=device)
                arrays.j = self.j.data_ptr()
        if "S" in quantities:
            self.shifts = torch.empty((n_pairs, 3), dtype=torch.int32, device=device)
            arrays.shifts = self.shifts.data_ptr()
        if "d" in quantities:
            self.distances = torch.empty(n_pairs, dtype=self.value_dtype, device=device)
            arrays.distances = self.distances.data_ptr()
        if "D" in quantities:
            self.vectors = torch.empty((n_pairs, 3), dtype=self.value_dtype, device=device)
            arrays.vectors = self.vectors.data_ptr()
        arrays.capacity = n_pairs

    def take(self, n_pairs):
        """The quantities in the order asked for, `n_pairs` rows each."""
        if n_pairs == 0 and self.arrays.capacity == 0:
            self.allocate(0)
        capacity = self.arrays.capacity
        # What a tensor holds on to, and what is written when it is saved, is its whole storage: an
        # eighth and 128 rows more than its own at most, or it is copied
        wasteful = capacity > n_pairs + n_pairs // 8 + 128

        result = []
        for k, quantity in enumerate(self.quantities):
            if quantity == "i":
                tensor = self.i
            elif quantity == "j":
                tensor = self.j
            elif quantity == "S":
                tensor = self.shifts
            elif quantity == "d":
                tensor = self.distances
            elif quantity == "D":
                tensor = self.vectors
            elif quantity == "P":
                tensor = self.pairs
            else:
                continue
            if tensor is None:  # an index beside the pairs
                result.append(self.pairs[:n_pairs, "ij".index(quantity)].clone())
                continue
            if capacity != n_pairs:
                tensor = tensor[:n_pairs]
                if wasteful:
                    tensor = tensor.clone()
            # a quantity asked for twice comes back as two tensors
            result.append(tensor.clone() if quantity in self.quantities[:k] else tensor)
        return result
