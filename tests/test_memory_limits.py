"""Calls that find no device memory return an error, keep what the context had, and
leave nothing behind: the next calls give what an undisturbed context gives, bit for
bit.  The memory is taken by allocations of the test's own, and given back."""
import ctypes

import numpy as np
import pytest

from tests.helpers import perturbed
from wcns_b200 import cases

pytestmark = pytest.mark.gpu

STATE = ("r", "u", "v", "w", "p")


class Hog:
    """Device memory taken down to `leave` bytes (0: whatever the allocator still gives)."""

    def __init__(self, leave=0):
        import torch
        self.rt = ctypes.CDLL("libcudart.so.12")
        self.rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
        self.rt.cudaFree.argtypes = [ctypes.c_void_p]
        self.held = []
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        top = torch.cuda.mem_get_info()[0] - leave
        size = 1 << 36
        while size >= (512 if leave == 0 else 1 << 21):
            if leave and size > top:
                size >>= 1
                continue
            p = ctypes.c_void_p()
            if self.rt.cudaMalloc(ctypes.byref(p), size) == 0:
                self.held.append(p)
                top -= size
            else:
                self.rt.cudaGetLastError()
                size >>= 1

    def __enter__(self):
        return self

    def __exit__(self, *a):
        for p in self.held:
            self.rt.cudaFree(p)


def _check(g, ref):
    np.testing.assert_array_equal(g.step(2), ref.step(2))
    for nb in range(1, len(g.dims) + 1):
        for f in STATE:
            np.testing.assert_array_equal(g.get(f, nb), ref.get(f, nb))


def test_line_tables_without_memory():
    from wcns_b200.solver import Wcns, WcnsError
    case = perturbed(cases.small_plate_case())
    g, ref = Wcns(case), Wcns(case)
    g.step(1), ref.step(1)
    shape = g.shape
    with Hog():
        for lines in (2, 3):
            with pytest.raises(WcnsError):
                g.set_shape(shape[:2] + [lines, lines])
            assert g.shape == shape
    _check(g, ref)
    g.set_shape(shape[:2] + [2, 2])  # with memory it is taken
    _check(g, ref)
