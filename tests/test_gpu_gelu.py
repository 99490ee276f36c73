"""The layers' BF16 GELU over every float: the approximation with its interval
and the reference decision give the reference's bits, and it decides by itself
for all but a small part of what the layers see."""
import ctypes as ct

import pytest

from anacor_public_gb300 import _lib, build

pytestmark = pytest.mark.gpu


def test_every_float_rounds_as_the_reference():
    build.build()
    L = _lib.load()
    wrong, opened = ct.c_uint64(), ct.c_uint64()
    assert L.anacor_gelu_check(ct.byref(wrong), ct.byref(opened)) == 0, _lib.last_error(L)
    assert wrong.value == 0
    # floats below about -4 (a quarter of all exponents there are) and few others
    assert opened.value < 0.26 * 2 ** 32
