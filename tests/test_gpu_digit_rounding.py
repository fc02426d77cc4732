"""Digit products at the worst digits of their dropped levels, and where the sum leaves the range
that is rounded without branches, against exact integers."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact(A, B):
    return [[sum((Fraction(a) * Fraction(b) for a, b in zip(r, c)), Fraction(0)) / 2 for c in B.T] for r in A]


def test_dropped_levels_at_their_worst(ccx):
    """Entries of digits (64, -128, ..., -128) beside a maximum of 1/2: all dropped pairs have one
    sign and their largest size (-x has other digits: none is +128).  Within 2^-51 of K max|A| max|B|, and the rounding of the result."""
    K = 1500
    x = 0.5 - sum(2.0 ** (-8 * i) for i in range(1, 7))
    A, B = np.full((2, K), x), np.full((K, 16), x)
    A[:, 0] = B[0] = 0.5
    A[1] = -A[1]
    C, want = ccx.selftest_tc_product(A, B, kind=2), exact(A, B[:, :1])
    for m in range(2):
        off = abs(Fraction(C[m, 0]) - want[m][0])
        assert off <= Fraction(K, 4 * 2 ** 52) + abs(want[m][0]) / 2 ** 53, float(off)
    assert np.array_equal(C, np.repeat(C[:, :1], 16, axis=1))


def test_sums_below_the_scale_of_their_row(ccx):
    """Two large products that cancel leave a sum below 2^-46 of the scale: exact, either sign."""
    t = np.array([3.0 * 2.0 ** -46, -5.0 * 2.0 ** -47, 2.0 ** -44, 0.0])
    A = np.stack([np.ones(4), -np.ones(4), t], axis=1)
    B = np.repeat(np.array([[1.0], [1.0], [2.0 ** -5]]), 16, axis=1)
    assert np.array_equal(ccx.selftest_tc_product(A, B, kind=2), np.repeat(t[:, None] * 2.0 ** -6, 16, axis=1))


@pytest.mark.parametrize("scale", [-530, -525, -519])
def test_subnormal_results(ccx, scale):
    """Within the least number (rounded to FP64's 53 bits and then to what a subnormal holds)."""
    r = np.random.RandomState(5)
    A, B = np.ldexp(r.uniform(-1, 1, (5, 40)), scale), np.ldexp(r.uniform(-1, 1, (40, 16)), scale)
    C, want = ccx.selftest_tc_product(A, B, kind=2), exact(A, B)
    for m in range(5):
        for n in range(16):
            assert abs(Fraction(C[m, n]) - want[m][n]) <= Fraction(1, 2 ** 1074) + abs(want[m][n]) / 2 ** 53


def test_results_at_the_end_of_the_range(ccx):
    """The largest binade is reached, what lies beyond is infinite."""
    A = np.ldexp([[1.5], [-1.5], [1.5], [-1.5]], [[511], [511], [512], [512]])
    C = ccx.selftest_tc_product(A, np.full((1, 16), 2.0 ** 513), kind=2)
    top = np.ldexp(1.5, 1023)
    assert np.array_equal(C, np.repeat([[top], [-top], [np.inf], [-np.inf]], 16, axis=1))
