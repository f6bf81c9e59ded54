"""touch_pages, which backs the caller's output array while it is still being
computed, leaves every byte as it is: a call that fails has changed nothing, and
an output that shares memory with the inputs does not destroy them.  No GPU."""
import ctypes

import numpy as np
import pytest

from vca_gb300 import solver


@pytest.mark.parametrize("at,n", [(0, 0), (0, 1), (5, 1), (1, 4095), (0, 4096), (4095, 4097), (17, 40001)])
def test_bytes_stay(at, n):
    touch = getattr(solver.load(), "_ZN3vca11touch_pagesEPvm")  # vca::touch_pages(void*, size_t)
    touch.argtypes, touch.restype = [ctypes.c_void_p, ctypes.c_size_t], None
    a = np.random.default_rng(n).integers(1, 256, at + n + 4096, dtype=np.uint8)
    b = a.copy()
    touch(b.ctypes.data + at, n)
    np.testing.assert_array_equal(a, b)


def test_fresh_pages_are_backed():
    """Writing to 64 MB that touch_pages has seen takes no page faults any more."""
    import resource
    touch = getattr(solver.load(), "_ZN3vca11touch_pagesEPvm")
    touch.argtypes, touch.restype = [ctypes.c_void_p, ctypes.c_size_t], None
    a = np.empty(64 << 20, dtype=np.uint8)
    touch(a.ctypes.data, a.size)
    before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
    a[::4096] = 1
    assert resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before < 64
