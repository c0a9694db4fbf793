"""Division by a constant from its double-word reciprocal (madv_exact.cuh) for divisors far from 1:
dividends whose quotient nears the subnormal numbers or the largest one, on significands next to a
rounding boundary (madv_selftest_exact draws those), against the IEEE division bit for bit."""
import ctypes as C

import pytest

from maestroex_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


@pytest.mark.parametrize("y", [1.0e8 / 42, 1.2345678901234567e20, 9.8765432109876543e60, 1.7654321e250, 3.1415926535897e-95,
                               2.7182818e-250, 4.9e-300, 7.7e305])
def test_quotients_are_correctly_rounded(y):
    nfail = C.c_longlong(-1)
    capi.check(capi.lib().madv_selftest_exact(y, 1.0e-3, 1 << 24, C.byref(nfail), None))
    assert nfail.value == 0
