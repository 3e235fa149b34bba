"""The corrected product that stands for a division on the positivity fit's
substitution chain: q0 = a rd with the rounded reciprocal rd, then
q = fma(fma(-d, q0, a), rd, q0) (Markstein, IBM J. Res. Dev. 34(1), 1990),
evaluated here in exact rationals, each step rounded once, against a / d."""

from fractions import Fraction

import numpy as np


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def quotient(a, d):
    rd = 1.0 / d
    q0 = a * rd
    return fma(fma(-d, q0, a), rd, q0)


def test_quotient_is_the_rounded_one():
    """Diagonal entries are square roots above sqrt(1e-9), and the dividends sums
    of a few products of the same constraints: exponents within 2^+-60."""
    rng = np.random.default_rng(1)
    n = 30000
    d = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-16, 30, n)
    a = rng.uniform(-2.0, 2.0, n) * 2.0 ** rng.integers(-60, 60, n)
    d[:6] = [1.0, np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0), 3.0, 1.5, np.nextafter(1.0, 0.0)]
    a[::97] = 0.0
    a[5::101] = d[5::101] * 3.0
    wrong = [(x, y) for x, y in zip(a.tolist(), d.tolist()) if quotient(x, y) != x / y]
    assert not wrong, wrong[:3]
