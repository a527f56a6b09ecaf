"""The packed ray map and camera map (ht_math.cuh hy_map<TWICE, true>): the bits of the IEEE form on
random maps and rays, and where half of their entries are zeros of either sign."""
import ctypes
import os

import pytest

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "libht_selftest.so")


@pytest.mark.parametrize("zeros", [0, 1])
def test_packed_maps_are_bit_identical(built, zeros):
    fn = ctypes.CDLL(LIB).ht_selftest_raymap_packed
    fn.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_ulonglong)]
    out = (ctypes.c_ulonglong * 2)()
    assert fn(1 << 25, 99 + zeros, zeros, out) == 0
    assert out[0] == 1 << 26
    assert out[1] == 0, f"{out[1]} maps differ"
