"""The square and cube roots of the closure's training features (an FP32 root and Newton steps in FP64)
keep the precision of the FP64 functions: ark_selftest_division counts square roots more than 0.501 ulp
and cube roots more than 1 ulp from the exact root (FP64 sqrt and cbrt: 0.5 and 1), exact squares and
cubes whose root is not exact, and zeros, infinities and NaN that do not come back."""
import ctypes

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,seed", [(1, 3), (17, 4), (1 << 22, 5)])
def test_training_roots_keep_fp64_precision(ark, n, seed):
    bad = ctypes.c_longlong(-1)
    assert ark.lib().ark_selftest_division(n, seed, ctypes.byref(bad)) == 0
    assert bad.value == 0
