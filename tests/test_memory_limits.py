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
    """All device memory but `leave` bytes (0: all that the allocator gives): chunks of
    2 MB are set aside, the rest is taken, and the chunks are given back."""

    def __init__(self, leave=0):
        import torch
        self.rt = ctypes.CDLL("libcudart.so.12")
        self.rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
        self.rt.cudaFree.argtypes = [ctypes.c_void_p]
        self.held = []
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        aside = [self._take(2 << 20) for _ in range(leave // (2 << 20))]
        size = 1 << 36
        while size >= (2 << 20 if leave else 512):
            p = self._take(size)
            if p is None:
                size >>= 1
            else:
                self.held.append(p)
        for p in aside:
            self.rt.cudaFree(p)

    def _take(self, size):
        p = ctypes.c_void_p()
        if self.rt.cudaMalloc(ctypes.byref(p), size) == 0:
            return p
        self.rt.cudaGetLastError()
        return None

    def __enter__(self):
        return self

    def __exit__(self, *a):
        for p in self.held:
            self.rt.cudaFree(p)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


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


@pytest.mark.parametrize("form", ["clustered", "wide"])
def test_autotune_without_memory_for_another_form(form):
    """Room for the tuner's copy of dq, not for the other form's arrays (25 MB of the
    clustered sweeps, 12 MB of the wide ones): the form in use stays, with the arrays
    and the captured step that belong to it."""
    from wcns_b200.solver import Wcns, WcnsError
    case = perturbed(cases.vortex_case(ni=65, nj=24, nk=16))
    g, ref = Wcns(case), Wcns(case)
    if form == "clustered":
        for h in (g, ref):
            h.set_shape([8, 0] + h.shape[2:])
    assert g.sweep_mode() == form
    shape = g.shape
    g.step(1), ref.step(1)
    with Hog(leave=6 << 20):
        if form == "clustered":
            with pytest.raises(WcnsError):
                g.autotune(1)
            assert g.shape == shape
        else:  # the lines per CTA are tuned all the same
            g.autotune(1)
        assert g.sweep_mode() == form
    _check(g, ref)


def test_autotune_keeps_only_the_arrays_of_the_form_it_takes():
    from wcns_b200.solver import Wcns
    case = perturbed(cases.vortex_case(ni=600, nj=48, nk=36))
    g = Wcns(case)
    assert g.sweep_mode() == "wide"
    g.step(1)
    before = _free()
    g.set_shape([16, 0] + g.shape[2:])  # the clustered arrays are 745 MB, the wide ones 346
    g.step(1)
    assert before - _free() < 500 << 20
    g.autotune(1)
    assert before - _free() < (100 if g.sweep_mode() == "wide" else 500) << 20
    g.set_shape([0, 0] + g.shape[2:])
    assert before - _free() < 100 << 20


def test_a_context_that_finds_no_memory_leaves_none_taken():
    """Room for the field pool (281 MB), the residual's buffers (47) or the sweeps'
    records, but not for all of them and the metrics' (75): an error, the memory
    back, and no error left over for the next call of another context."""
    from wcns_b200.solver import Wcns, WcnsError
    small = perturbed(cases.small_plate_case())
    big = cases.vortex_case(ni=121, nj=75, nk=51)
    other, ref = Wcns(small), Wcns(small)
    other.step(1), ref.step(1)
    Wcns(big).close()  # what the library keeps from a first use is there
    before = _free()
    kept = Wcns(big)
    all_but_metrics = (before - _free() >> 20) + 40
    kept.close()
    for room in (40, 300, 360, all_but_metrics):
        with Hog(leave=room << 20):
            before = _free()
            with pytest.raises(WcnsError):
                Wcns(big)
            assert before - _free() < 8 << 20, room
        _check(other, ref)
    Wcns(big).close()
