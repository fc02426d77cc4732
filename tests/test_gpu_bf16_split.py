"""The BF16 split of FP64 operands, hi + lo, each rounded once to 8 bits (half away from zero):
values whose remainder lies at or one unit of FP64 beside the middle of two lows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def nearest8(m):
    """The integer m to 8 significant bits, halves away from zero, by integers."""
    a = abs(int(m))
    drop = max(a.bit_length() - 8, 0)
    a = ((a + (1 << drop >> 1)) >> drop) << drop
    return a if m >= 0 else -a


def test_both_halves_are_rounded_once(ccx):
    r = np.random.RandomState(4)
    x, want = [], []
    for i in range(3000):
        H, low, shift = r.randint(129, 256), r.randint(128, 256), r.randint(28, 36)
        R = ((2 * low + r.randint(0, 2)) << shift) + (i % 3 - 1 if i < 2400 else r.randint(-1000, 1000))
        M = ((H << 45) + (R if r.randint(2) else -R)) * (1 if r.randint(2) else -1)
        hi = nearest8(M)
        e = r.randint(-60, 20)
        x.append(np.ldexp(float(M), e))
        want.append(np.ldexp(float(hi + nearest8(M - hi)), e))
    # a product with 1 is hi + lo, which FP32 holds where lo begins within 16 bits of hi's end
    C = ccx.selftest_tc_product(np.array(x)[:, None], np.ones((1, 16)))
    assert np.array_equal(2.0 * C[:, 0], np.array(want))
