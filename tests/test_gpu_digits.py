"""Known answer of the instruction that the digit GEMMs use: sums of products of
8-bit digits, several digits of one operand in one MMA, are exact integers."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["stokes_gpu_selftest_tensor", "stokes_gpu_selftest_tma"])
def test_digit_sums_are_exact(lib, name):
    err = C.c_double(-1.0)
    assert getattr(lib, name)(C.byref(err)) == 0, lib.stokes_gpu_last_error_message().decode()
    assert err.value == 0.0
