"""The reciprocals that the fused substages form from the hardware estimates."""
import ctypes as C

import pytest

from mhd_gb300 import abi

pytestmark = pytest.mark.gpu


def test_reciprocals_within_their_error_bounds():
    """FP32, on every float: 2^-24 + 2^-43 of the value where the result is an
    ordinary number, the quotient's zeros, infinities and NaN, and subnormal
    numbers to a unit in the last place.  FP64, on 2^24 patterns over the
    exponents: 2^-53 + 2^-59."""
    bad32, bad64 = C.c_longlong(-1), C.c_longlong(-1)
    abi.check(abi.load().mhd_selftest_recip(1 << 24, 20261205, C.byref(bad32), C.byref(bad64)))
    assert (bad32.value, bad64.value) == (0, 0)
