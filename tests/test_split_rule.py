"""The rule of lanes per ray of a single render (152 SMs), at its edges: all
blocks resident at once, 4 or 5 per SM by the records, and 4 for the two lanes
of half records of fewer than 2^21 texels."""

import ctypes

import pytest

from pyvr_gb300 import _native

# (compact, texels): most blocks of 4 lanes and of 2 lanes
LIMITS = [((False, 1), (608, 608)), ((False, 1 << 21), (608, 608)),
          ((True, (1 << 21) - 1), (760, 608)), ((True, 1 << 21), (760, 760))]


@pytest.mark.parametrize("volume,most", LIMITS)
def test_split_lanes(volume, most):
    f = getattr(_native.load(), "_ZN3pvr11split_lanesEiiibx")
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_bool, ctypes.c_longlong]
    f.restype = ctypes.c_int
    four, two = most  # blocks of 8x8 and of 8x16 pixels, in one column
    for height, lanes in ((1, 4), (8 * four, 4), (8 * four + 1, 2), (16 * two, 2), (16 * two + 1, 1), (32768, 1)):
        assert f(8, height, 152, *volume) == lanes, height
    assert f(32768, 32768, 152, *volume) == 1
