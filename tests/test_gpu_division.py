"""The full energy's division by a constant equals IEEE division on every float of its range,
for the divisors of the device's own tables."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_constant_division(ctx, pkg):
    wrong = C.c_int64(-1)
    assert pkg.lib().binder_selftest_div(ctx._h, C.byref(wrong)) == 0
    assert wrong.value == 0
