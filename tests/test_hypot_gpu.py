"""hypot_fast (csrc/exact_math.cuh), the hypot of every TV-L1 iteration: its root
against the IEEE square root for every upper word the estimate can see, over the
exponents of sums of squares of floats, and its results against hypot_ref on
pairs of any size and on and next to the midpoints where rounding could part."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _count(of, which, lo, hi, seed=0):
    n = C.c_ulonglong(0)
    assert of.capi.lib().oflow_selftest_math(which, lo, hi, seed, C.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("exponent", [-400, -300, -146, -2, 0, 2, 24, 130, 256])
def test_root_within_its_units(of, exponent):
    k = (exponent + 400) // 2
    assert _count(of, 4, k << 21, (k + 1) << 21) == 0


def test_root_over_every_exponent(of):
    """Every 61st upper word, over all exponents in turn."""
    for k in range(0, 330, 3):
        lo = (k << 21) + 61 * k
        assert _count(of, 4, lo, lo + (1 << 15)) == 0


def test_the_count_counts(of):
    """The roots are not all the IEEE square roots (none is more than a unit away)."""
    assert _count(of, 4, 200 << 21, 201 << 21, 1) > 0
    assert _count(of, 4, 200 << 21, 201 << 21, 2) == 0


@pytest.mark.parametrize("seed", [11, 12])
def test_results_it_vouches_for(of, seed):
    assert _count(of, 5, 0, 1 << 28, seed) == 0
