"""The quotients that carry a proof instead of a check of their result
(exact_div.cuh), on the device: against its division operator bit for bit,
and the premise of the limiter's, the error of the reciprocal estimate."""
import ctypes as C

import pytest

from volcano_ash3d_b200 import _lib

pytestmark = pytest.mark.gpu


def test_quotients_are_ieee():
    lib = _lib.load()
    n = 1 << 26
    counts, estimate = (C.c_uint64 * 4)(), C.c_double(1.0)
    _lib.check(lib.a3g_selftest_quotients(0, n, 2718, counts, C.byref(estimate)))
    assert counts[0] == 0 and counts[1] == 0
    # most pairs take the fast way: of the ratios 20 exponents in 420, of the dividends the tails below 2^-900 (17 in
    # 109 of a quarter), and of either the divisors just below a power of two (five in sixteen of two families) do not
    assert counts[2] < 0.4 * n and counts[3] < 0.4 * n
    assert 0.0 < estimate.value < 2.0**-19
