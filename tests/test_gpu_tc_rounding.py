"""How the correction products' accumulators become FP64: operands with one non-zero term an
accumulator, so that what is added is known exactly (three accumulators of 64 columns each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sums(ccx, terms, scale=0, n=17):
    """1/2 of the sum of three accumulators that hold terms[m] 2^(2 scale)."""
    A, B = np.zeros((len(terms), 192)), np.zeros((192, n))
    A[:, ::64] = np.ldexp(terms, scale)
    B[::64] = np.ldexp(1.0, scale)
    C = ccx.selftest_tc_product(A, B, segments=True)
    assert np.array_equal(C, np.repeat(C[:, :1], n, axis=1), equal_nan=True)
    return C[:, 0]


def test_sums_of_two_accumulators_are_rounded_once(ccx):
    """Two terms of 16 bits (exact as BF16 pairs) with either sign and up to 2^50 apart: their FP64
    sum, to one unit in the last place where more than 53 bits are needed, exact otherwise.  Powers
    of two with a small term of the other sign end in the binade below."""
    r = np.random.RandomState(2)
    a = np.ldexp(r.randint(1 << 15, 1 << 16, 500).astype(float), r.randint(-30, 30, 500)) * r.choice([-1.0, 1.0], 500)
    a[:100] = np.ldexp(1.0, r.randint(-20, 20, 100)) * r.choice([-1.0, 1.0], 100)
    b = np.ldexp(r.randint(1 << 15, 1 << 16, 500).astype(float), r.randint(-50, 30, 500)) * r.choice([-1.0, 1.0], 500)
    b[400:] = -a[400:]  # cancels
    got, want = 2.0 * sums(ccx, np.stack([a, 0 * a, b], axis=1)), a + b
    exact = want.astype(np.longdouble) == a.astype(np.longdouble) + b.astype(np.longdouble)
    assert np.array_equal(got[exact], want[exact]) and exact.sum() > 100
    assert np.all(np.abs(got - want) <= np.spacing(np.abs(want)))


@pytest.mark.parametrize("scale", [-74, -60, 61])
def test_sums_outside_the_range_of_fp32_pairs(ccx, scale):
    """Accumulators whose sum passes the FP32 range (each of them below it), or whose rounding is
    subnormal: the FP64 sum of the three.  Subnormal accumulators may be held as they are or as
    zeros; added as eighths, each of three rounds by half of 2^-149, eightfold: within 2^-145."""
    t = np.array([[40.0, 50.0, 45.0], [-60.0, -33.0, -61.0], [63.0, -62.0, 63.0], [1.0, 0.125, -3.0], [3.0, 0.0, 0.0]])
    if scale < 0:
        t = np.concatenate([t, [[2.0 ** 20, 0.0, 1.0 + 2.0 ** -15], [-2.0 ** 20, 1.0 + 2.0 ** -15, -1.5]]])
    got, want = sums(ccx, t, scale), 0.5 * np.ldexp(t.sum(axis=1), 2 * scale)
    assert np.all(np.abs(got - want) <= (0.0 if scale > -64 else np.abs(want) + 2.0 ** -145)), (got, want)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_infinities_and_nans_stay(ccx, bad):
    got = sums(ccx, np.array([[1.0, bad, 2.0], [1.0, 1.0, 2.0]]))
    assert not np.isfinite(got[0]) and got[1] == 2.0
