"""The solve's quotient from a correctly rounded reciprocal (chol_div in tdi_cholesky.cuh) against the
correctly rounded division, with every operation restated exactly (fractions rounded once to double):
random operands, divisors with extreme mantissas and quotients next to rounding boundaries."""
from fractions import Fraction

import numpy as np


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def chol_div(t, l):
    r = float(Fraction(1) / Fraction(l))
    q0 = t * r
    q1 = fma(fma(-q0, l, t), r, q0)
    return fma(fma(-q1, l, t), r, q1)


def test_quotient_is_correctly_rounded():
    rng = np.random.default_rng(4)
    n = 0
    for i in range(20000):
        l = float(rng.uniform(1, 2) * 2.0 ** rng.integers(-60, 60))
        if i % 4 == 1:                                  # mantissa near all ones or one
            l = float(np.ldexp(2.0 - 2.0 ** -52 * rng.integers(1, 6), int(rng.integers(-20, 20))))
        elif i % 4 == 2:
            l = float(np.ldexp(1.0 + 2.0 ** -52 * rng.integers(0, 6), int(rng.integers(-20, 20))))
        t = float(rng.normal() * 2.0 ** rng.integers(-200, 200))
        if i % 2:                                       # quotients beside a midpoint between two doubles
            q = float(rng.uniform(1, 2))
            t = float((Fraction(q) + Fraction(int(rng.integers(0, 2)) * 2 - 1, 2 ** 53)) * Fraction(l))
        if t == 0.0:
            continue
        assert chol_div(t, l) == t / l, (t, l)
        n += 1
    assert n > 19000
