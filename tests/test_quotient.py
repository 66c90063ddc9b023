"""The solvers' fast quotient (solve_common.cuh quot_fast): a / D from y = RN(1 / D) by
q0 = RN(a y), e = RN(q0 D - a), q = RN(q0 - e y). Only quotients next to a rounding boundary can
come out wrong, so it is checked on those, in exact arithmetic: with significands a = A 2^-23
and D = B 2^-23, the boundaries nearest to a / D are M / 2^s with M odd (s = 24 where A >= B,
else 25), and A 2^s - M B = N is small for the quotients nearest to them.
"""
from fractions import Fraction

import numpy as np
import pytest


def rn(v: Fraction) -> Fraction:
    """v to the nearest 24-bit significand, ties to even (no exponent range)."""
    if v == 0:
        return v
    s, v = (-1 if v < 0 else 1), abs(v)
    e = v.numerator.bit_length() - v.denominator.bit_length() - 24
    while v / Fraction(2) ** e >= 2 ** 24:
        e += 1
    while v / Fraction(2) ** e < 2 ** 23:
        e -= 1
    m = v / Fraction(2) ** e
    k = m.numerator // m.denominator
    r = m - k
    if r > Fraction(1, 2) or (r == Fraction(1, 2) and k & 1):
        k += 1
    return s * k * Fraction(2) ** e


def quot_fast(a: Fraction, d: Fraction) -> Fraction:
    y = rn(1 / d)
    q0 = rn(a * y)
    return rn(q0 - rn(q0 * d - a) * y)


@pytest.mark.parametrize("seed", range(4))
def test_quotients_next_to_a_rounding_boundary(seed):
    rng = np.random.default_rng(seed)
    checked = 0
    for _ in range(400):
        B = int(rng.integers(2 ** 22, 2 ** 23)) * 2 + 1   # odd, so that it has an inverse modulo 2^s
        for s in (24, 25):
            for N in (-3, -1, 1, 3):
                M = (-N * pow(B, -1, 2 ** s)) % 2 ** s
                A, r = divmod(M * B + N, 2 ** s)
                if r or not M & 1 or not 2 ** 23 <= A < 2 ** 24 or (A >= B) != (s == 24):
                    continue
                a, d = Fraction(A, 2 ** 23), Fraction(B, 2 ** 23)
                assert quot_fast(a, d) == rn(a / d), (A, B)
                assert quot_fast(-a * 2 ** 31, d / 2 ** 20) == rn(-a / d * 2 ** 51)
                checked += 1
    assert checked > 200
