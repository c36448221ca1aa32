"""Sizes the group quantiser refuses, by its return code and before anything is launched."""
import ctypes as C

from ateniaengine_b200 import _lib

ERR_SHAPE = -2


def test_more_than_four_times_two_to_the_31_scales_are_refused():
    lib = _lib.lib()
    p = C.c_void_p(16)  # never read: the call returns before it launches
    for K, N, g in [(100_000, 100_000, 1), (1 << 17, 1 << 17, 1), (1 << 20, 1 << 16, 4)]:
        assert -(-K // g) * N > 4 * 0x7FFFFFFF
        assert lib.atenia_quantize_per_group_i8(p, K, N, g, p, p, None) == ERR_SHAPE
