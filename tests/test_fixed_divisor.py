"""Division by a divisor known in advance, in two FP64 operations from its
reciprocal in two words (divide.cuh, div2 and div_class), restated in exact
rational arithmetic: a divisor of class 0 gives the correctly rounded quotient
for every numerator, one of class 1 after one Markstein correction.
"""
import random
from fractions import Fraction

import pytest

ONE = 1 << 52


def rn(x):
    return x.numerator / x.denominator   # int / int is correctly rounded


def fma(a, b, c):
    return rn(Fraction(a) * Fraction(b) + Fraction(c))


def words(b):
    yh = rn(1 / Fraction(b))
    return yh, rn(1 / Fraction(b) - Fraction(yh))


def div2(a, yh, yl):
    return fma(a, yh, a * yl)


def critical(B):
    """The numerators whose quotients come closest to a midpoint."""
    if B % 2 == 0:
        return []
    x = pow(pow(2, 54, B), -1, B)
    return [A for A in (x, B - x) if A >= ONE]


def div_class(B):
    b = B / ONE
    yh, yl = words(b)
    return int(any(div2(A / ONE, yh, yl) != rn(Fraction(A, B)) for A in critical(B)))


def quotient(a, b, cls):
    yh, yl = words(b)
    q = div2(a, yh, yl)
    if cls:
        q = fma(fma(-q, b, a), yh, q)
    return q


@pytest.mark.parametrize('seed', range(4))
def test_quotients(seed):
    rng = random.Random(seed)
    special = [ONE, ONE + 1, 2 * ONE - 1, 2 * ONE - 2, 2 * ONE - 3, 3 << 51, (3 << 51) + 1]
    classes = set()
    for _ in range(400):
        B = rng.choice(special) if rng.random() < 0.2 else rng.randrange(ONE, 2 * ONE)
        cls = div_class(B)
        classes.add(cls)
        As = critical(B) + [rng.randrange(ONE, 2 * ONE) for _ in range(6)] + [ONE, 2 * ONE - 1, B, min(B + 1, 2 * ONE - 1)]
        for A in As:
            assert quotient(A / ONE, B / ONE, cls) == rn(Fraction(A, B)), (A, B, cls)
    assert 0 in classes


def test_the_correction_is_needed_for_some_divisors():
    """Divisors whose critical numerator rounds wrongly in two operations
    exist, and the correction mends them."""
    rng = random.Random(7)
    found = 0
    for _ in range(4000):
        B = rng.randrange(ONE, 2 * ONE) | 1
        if div_class(B):
            found += 1
            for A in critical(B):
                assert quotient(A / ONE, B / ONE, 1) == rn(Fraction(A, B))
    assert found > 0
