"""The setup's FP64 fixed-point product up to the end of its range, |a b| 2^sc < 2^63, against exact rationals."""
import random
from fractions import Fraction

from test_fixed_product import fixed  # noqa: F401  (the header's function compiled for the host)


def test_top_bit(fixed):  # noqa: F811
    rng = random.Random(9)
    n = 0
    for _ in range(4000):
        a = rng.uniform(-1.0, 1.0) * 2.0 ** rng.randint(-300, 300)
        b = rng.uniform(-1.0, 1.0) * 2.0 ** rng.randint(-300, 300)
        p, sc = abs(Fraction(a) * Fraction(b)), 0
        if not p:
            continue
        sc = 62 - (p.numerator.bit_length() - p.denominator.bit_length())
        while p * Fraction(2) ** sc >= Fraction(2) ** 63 - 1:
            sc -= 1
        while p * Fraction(2) ** (sc + 1) < Fraction(2) ** 63 - 1:
            sc += 1
        exact = Fraction(a) * Fraction(b) * Fraction(2) ** sc
        assert 2 ** 61 < abs(exact) < 2 ** 63
        assert fixed(a, b, sc) == round(exact)
        n += 1
    assert n > 3000
