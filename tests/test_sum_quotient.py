"""The quotients of sums that alpha and beta of the one-launch solve are: the nearest FP32 number to the quotient of the
exact sums of FP32 values, as FP64 sums give it, for any number of values, any range and quotients close to the middle
between two FP32 numbers.  Expected values by rational arithmetic."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu


def _quotients(a, b, exact):
    f = L.lib().amr_test_sum_quotient
    f.argtypes = [C.c_int64, C.c_int32, C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p]
    a, b = np.ascontiguousarray(a, np.float32), np.ascontiguousarray(b, np.float32)
    out = np.zeros(len(a), np.float32)
    assert f(len(a), a.shape[1], L.ptr(a), L.ptr(b), exact, L.ptr(out)) == 0
    return out


def _nearest(a, b):
    """FP64 nearest, then FP32: the same as FP32 nearest for quotients not within 2^-54 of the middle, as all here."""
    out = []
    for x, y in zip(a, b):
        out.append(np.float32(float(sum(map(Fraction, x.tolist())) / sum(map(Fraction, y.tolist())))))
    return np.array(out, np.float32)


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("n", [1, 16, 31, 33, 51, 64, 100, 128, 200, 256, 300, 512])
def test_values_over_many_magnitudes(n, exact):
    rng = np.random.default_rng(n)
    cases = max(40, 4000 // n)
    a = np.exp(rng.normal(0, 4, (cases, n))) * rng.normal(0, 1, (cases, n)) ** 2 * np.exp(rng.normal(0, 10, (cases, 1)))
    b = np.exp(rng.normal(0, 4, (cases, n))) * np.abs(rng.normal(0, 1, (cases, n)))
    b[:, ::7] *= np.where(rng.random((cases, 1)) < 0.5, -0.01, 1.0)  # some sums with terms of either sign
    b[:, 0] += 2 * np.abs(b).sum(axis=1)
    a, b = a.astype(np.float32), b.astype(np.float32)
    assert np.array_equal(_quotients(a, b, exact), _nearest(a, b))


@pytest.mark.parametrize("exact", [0, 1])
def test_quotients_beside_the_middle_of_two_numbers(exact):
    """a = (q + half an ulp) b, exactly as a sum, and a term that moves the quotient off the middle by 2^-47 to 2^-50."""
    rng = np.random.default_rng(3)
    rows_a, rows_b = [], []
    for _ in range(400):
        q = Fraction(int(rng.integers(2 ** 23, 2 ** 24)) * 2 + 1, 2 ** 25)       # 25 bits: the middle of two
        b = [int(v) for v in rng.integers(2 ** 20, 2 ** 24, 40)]
        a = q * sum(b)
        terms, rest = [], a * 2 ** 25
        assert rest.denominator == 1
        rest = int(rest)
        while rest:  # parts of 24 bits
            low = rest & (2 ** 24 - 1)
            terms.append(Fraction(low, 1))
            rest >>= 24
        vals = [float(t) * 2.0 ** (24 * i - 25) for i, t in enumerate(terms)]
        off = float(a) * 2.0 ** -int(rng.integers(47, 51)) * (1 if rng.random() < 0.5 else -1)
        vals = vals + [float(np.float32(off))]
        rows_a.append(vals + [0.0] * (40 - len(vals)))
        rows_b.append([float(v) for v in b])
    a, b = np.array(rows_a, np.float32), np.array(rows_b, np.float32)
    assert np.array_equal(a.astype(np.float64), np.array([[np.float32(v) for v in r] for r in rows_a], np.float64))
    assert np.array_equal(_quotients(a, b, exact), _nearest(a, b))


@pytest.mark.parametrize("power", [-120, -60, 60, 110])
def test_ranges(power):
    rng = np.random.default_rng(5)
    a = np.abs(rng.normal(1, 1, (200, 51))).astype(np.float32) * np.float32(2.0 ** power)
    b = np.abs(rng.normal(1, 1, (200, 51))).astype(np.float32) * np.float32(2.0 ** power)
    for exact in (0, 1):
        assert np.array_equal(_quotients(a, b, exact), _nearest(a, b))


def test_zero_infinite_and_nan():
    a = np.array([[0.0, 0.0], [1.0, 2.0], [1.0, np.nan], [1.0, 2.0], [np.inf, 1.0]], np.float32)
    b = np.array([[1.0, 2.0], [0.0, 0.0], [1.0, 2.0], [np.inf, 1.0], [1.0, 2.0]], np.float32)
    out = _quotients(a, b, 0)
    assert out[0] == 0 and np.isnan(out[1]) and np.isnan(out[2]) and out[3] == 0 and np.isinf(out[4])
