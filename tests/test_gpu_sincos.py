"""The hemisphere sampler's sine and cosine (ht_math.cuh: sincos_turn): equal to CUDA's FP64 sincos
rounded to float at the angle of every 32-bit RNG state, and the half turn of rot3_look_at a
constant of the same value."""
import ctypes
import os
import struct

import pytest

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "libht_selftest.so")


def _call(name):
    out = (ctypes.c_ulonglong * 2)()
    fn = getattr(ctypes.CDLL(LIB), name)
    fn.argtypes = [ctypes.POINTER(ctypes.c_ulonglong)]
    assert fn(out) == 0
    return out[0], out[1]


def test_sincos_turn_equals_fp64_at_every_state(built):
    checked, mismatches = _call("ht_selftest_sincos")
    assert checked == 1 << 32
    assert mismatches == 0


def test_half_turn_constants(built):
    sine, cosine = (struct.unpack("<f", struct.pack("<I", v))[0] for v in _call("ht_selftest_half_turn"))
    assert sine == 1.0 and cosine == float.fromhex("-0x1.777a5cp-25")
