"""Arithmetic that the kernels rest on and no specification promises, checked on
the device.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units", [(0, 0), (8, 8), (10, 12), (64, 64)])
def test_far_units_agree_with_bins(gpu_ctx, units):
    """The far kernel works on distances scaled by 2^-24, the near kernel and the
    fix-up on distances in bins: the same floats, guard bins and flags for every
    squared distance from 1 to 2^32 bins^2 (512 A).  The guard's multipliers are
    1 -/+ a few units of 2^-24."""
    from autogrid_b200 import load_library
    bad = (C.c_int64 * 3)()
    lo, hi = 1.0 - units[0] * 2.0 ** -24, 1.0 + units[1] * 2.0 ** -24
    assert load_library().ag_diag_far_units(0, 0, 32, lo, hi, bad) == 0
    assert list(bad) == [0, 0, 0]


def test_roots(gpu_ctx):
    """The FP32 root is the correctly rounded one everywhere.  The FP64
    reciprocal root is within 1.6 * 2^-53: x y rounded moves e = 1 - x y^2 by
    2^-53 and the result by half of that, the last operation rounds by 2^-53,
    and the seed's error of at most 2^-20 leaves (5/16) (2^-19)^3."""
    from autogrid_b200 import load_library
    bad, ulps = C.c_int64(), C.c_double()
    assert load_library().ag_diag_root_errors(0, C.byref(bad), -80, 64, C.byref(ulps)) == 0
    assert bad.value == 0
    assert 0.0 < ulps.value <= 1.6, ulps.value
