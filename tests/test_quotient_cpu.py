"""The refinement step of quotient_127 (mlops_b200/csrc/kernels/fbla_device.cuh) in exact integer arithmetic: from every
approximate reciprocal within 1 ulp it ends in the correctly rounded 127 / a, for every a of 16 significand bits."""
from fractions import Fraction

import pytest


def _round24(x):
    """x > 0 rounded to 24 significand bits, ties to even"""
    e = x.numerator.bit_length() - x.denominator.bit_length()
    if Fraction(2) ** e > x:
        e -= 1
    ulp = Fraction(2) ** (e - 23)
    n, rest = divmod(x, ulp)
    n = int(n) + (rest * 2 > ulp or (rest * 2 == ulp and n % 2 == 1))
    return n * ulp, ulp


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_refined_quotient_is_correctly_rounded(ulps):
    for m in range(1 << 15, 1 << 16, 1 if ulps else 3):
        a = Fraction(m)
        r, ulp = _round24(1 / a)
        r += ulps * ulp
        q0, _ = _round24(127 * r)
        e = 127 - a * q0
        assert e == 0 or abs(_round24(abs(e))[0]) == abs(e), m  # the residual is a float: the FMA that forms it does not round
        assert _round24(q0 + e * r)[0] == _round24(127 / a)[0], m
