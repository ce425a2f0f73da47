"""The integer forms of FP64 products and of conversions between FP32 and FP64, on the device against the
device's own instructions bit for bit (ark_selftest_division counts differences): ties of the rounding,
exponents at the edges of the range taken, zeros, subnormals, overflow, infinities and NaN."""
import ctypes

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,seed", [(1, 1), (33, 2), (1 << 24, 3), (1 << 24, 2**63 + 4)])
def test_integer_products_and_conversions_match_the_instructions(ark, n, seed):
    bad = ctypes.c_longlong(-1)
    assert ark.lib().ark_selftest_division(n, seed, ctypes.byref(bad)) == 0
    assert bad.value == 0
