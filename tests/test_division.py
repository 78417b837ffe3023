"""The short division of the probability passes (csrc/rs_common.cuh, div_by): the rounded reciprocal, a product and two
fused corrections give the correctly rounded quotient (Markstein 1990).  The steps are repeated here in exact rational
arithmetic, rounded to fp32 after every one, on random operands and on operands next to rounding midpoints."""
from fractions import Fraction

import numpy as np


def rn(x):
    """Fraction -> nearest fp32 (ties to even), normal range."""
    if x == 0:
        return np.float32(0)
    s, x = (-1, -x) if x < 0 else (1, x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    if Fraction(2) ** e > x:
        e -= 1
    ulp = Fraction(2) ** (max(e, -126) - 23)
    n, r = divmod(x, ulp)
    n = int(n) + (1 if (r > ulp / 2 or (r == ulp / 2 and int(n) % 2)) else 0)
    return np.float32(s * float(n * ulp))


def fma(a, b, c):
    return rn(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


def div_by(a, b, y):
    q = rn(Fraction(float(a)) * Fraction(float(y)))
    for _ in range(2):
        r = fma(-q, b, a)
        assert r == 0 or abs(r) >= np.float32(2.0 ** -126), (a, b)      # no remainder is subnormal
        q = fma(r, y, q)
    return q


def test_two_corrections_give_the_rounded_quotient():
    g = np.random.default_rng(3)
    for i in range(3000):
        b = np.float32(np.exp2(g.uniform(0, 20)))
        if i % 3 == 0:                       # all-ones significands: the reciprocal's error is largest here
            b = np.nextafter(np.float32(2.0 ** g.integers(1, 20)), np.float32(0))
        y = rn(1 / Fraction(float(b)))
        if i % 2:                            # next to a midpoint of two neighbouring quotients
            m = Fraction(float(np.float32(np.exp2(g.uniform(-60, -20))))) * (1 + Fraction(1, 2 ** 24))
            a = rn(m * Fraction(float(b)))
        else:
            a = np.float32(2.0 ** -78) if i % 50 == 0 else np.float32(np.exp2(g.uniform(-78, 0)))      # down to kDivMin
        assert a >= np.float32(2.0 ** -78)
        assert div_by(a, b, y) == rn(Fraction(float(a)) / Fraction(float(b))), (a, b)
