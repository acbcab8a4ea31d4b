"""The bounds of the fixed-point transforms' plans, for every length that a row or a column can have:
moduli below 2^62 from the input on, and below 2^63 after the values are scaled up on the way."""
import ctypes as C
import math
from fractions import Fraction

import pytest


def _lengths():
    def smooth(n):
        for p in (2, 3, 5, 7):
            while n % p == 0:
                n //= p
        return n == 1
    return [n for n in range(2, 2049) if smooth(n)]


def _growth(i, p):
    """Bound of a stage's growth of the moduli: twiddled butterflies of radix 3, 4, 5, 7 divide by 4"""
    return Fraction(p, 4) if i and p > 2 else Fraction(p)


@pytest.mark.parametrize("narrow", [0, 1])
def test_plans_of_every_length(lib, narrow):
    scaled = []
    for n in _lengths():
        radix, head, renorm = (C.c_int * 8)(), C.c_int(), C.c_int()
        ns = lib.kc_transform_plan(n, narrow, radix, C.byref(head), C.byref(renorm))
        assert 2 <= ns <= 8 and math.prod(radix[:ns]) == n
        # squares of moduli: components of 2^b make a modulus of sqrt(2) 2^b
        at, peak = Fraction(1), Fraction(1)
        for i in range(ns):
            at *= _growth(i, radix[i])
            peak = max(peak, at)
        assert 2 * (peak * Fraction(2) ** (62 - head.value)) ** 2 <= Fraction(2) ** 124, n
        if not renorm.value:
            assert n <= 256 and not narrow or ns < 4 or n == 686
            continue
        scaled.append(n)
        # stage 1 is the first whose outputs are looked at, and the last stage does not scale
        assert 2 <= renorm.value <= ns - 2, n
        at, peak = Fraction(1), Fraction(1)
        for i in range(renorm.value, ns):
            at *= _growth(i, radix[i])
            peak = max(peak, at)
        assert 2 * (peak * Fraction(2) ** 61) ** 2 < Fraction(2) ** 126 * Fraction(99, 100), n
    assert {288, 320, 512, 1024, 1440, 2048} <= set(scaled) and 343 not in scaled and 686 not in scaled


def test_lengths_without_a_plan(lib):
    radix, v = (C.c_int * 8)(), [C.c_int() for _ in range(2)]
    for n in (0, 1, 11, 22, 26, 1331):
        assert lib.kc_transform_plan(n, 0, radix, *map(C.byref, v)) == -1
