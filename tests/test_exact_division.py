"""The three-operation quotient of exact_div.cuh at small precisions: RN(a y), the remainder, the correction, against
RN(a / b) for every pair of significands, with the reciprocal y = RN(1 / b) (and so its error of up to half a unit)."""
from fractions import Fraction

import pytest


def _rn(x, p):
    """x rounded to p significant bits, ties to even."""
    if x == 0:
        return Fraction(0)
    n, d = abs(x).numerator, abs(x).denominator
    e = n.bit_length() - d.bit_length() - p
    while Fraction(n, d) >= Fraction(2) ** (p + e):
        e += 1
    while Fraction(n, d) < Fraction(2) ** (p + e - 1):
        e -= 1
    unit = Fraction(2) ** e
    m, rem = divmod(Fraction(n, d), unit)
    if 2 * rem > unit or (2 * rem == unit and m % 2):
        m += 1
    return (1 if x > 0 else -1) * m * unit


@pytest.mark.parametrize("p", [4, 5, 6, 7])
def test_quotient_is_correctly_rounded(p):
    lo, hi = 2 ** (p - 1), 2 ** p
    for b in range(lo, hi):
        y = _rn(Fraction(1, b), p)
        for a in range(lo, hi):
            q0 = _rn(a * y, p)
            r = _rn(b * q0 - a, p)
            assert _rn(q0 - r * y, p) == _rn(Fraction(a, b), p), (a, b)
