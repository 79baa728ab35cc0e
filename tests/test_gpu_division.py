"""The step kernels' shorter divisions (ndiv, cdiv of ecogen_b200/csrc/ecg_ieee.cuh) against CUDA's correctly
rounded a / b on hashed operands, special values and all-ones-significand divisors included: the quotients
are equal but for the two cases the header names (sign of a zero quotient over a negative divisor, a power
of two over an all-ones significand)."""
import ctypes as C
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROBE = os.path.join(ROOT, "ecogen_b200", "libecg_probe.so")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emin,emax", [(0, 0), (-4, 4), (-60, 60), (-500, 500)])
def test_step_divisions_equal_ieee_quotients(emin, emax):
    lib = C.CDLL(PROBE)
    lib.ecg_probe_division_check.argtypes = [C.c_ulonglong, C.c_int, C.c_int, C.c_int, C.c_int,
                                             C.POINTER(C.c_ulonglong)]
    counts = (C.c_ulonglong * 3)()
    assert lib.ecg_probe_division_check(0xD1710000 + emax, emin, emax, 148 * 8, 256, counts) == 0
    assert counts[0] == 148 * 8 * 256 * 256
    assert counts[1] == 0, f"{counts[1]} of {counts[0]} ndiv quotients differ"
    assert counts[2] == 0, f"{counts[2]} of {counts[0]} cdiv quotients differ"
