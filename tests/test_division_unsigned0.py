"""The exact division of the FP64 pair, matrix and cell arithmetic
(div_rn_unsigned0, sph_kernels.cu), restated on the CPU: div_rn without its two
tests for a zero remainder,
    q0 = RN(a y); q1 = RN(q0 + RN(a - b q0) y); q = RN(q1 + RN(a - b q1) y)
with y = RN(1/b).  It is the IEEE quotient bit for bit except that -0 over a
positive divisor gives +0, which its callers rule out or add to +0."""
import math
from fractions import Fraction

from tests.test_division_method import _bits, _operands


def _fma(x, y, z):
    """RN(x y + z) with the sign of a zero as IEEE 754 has it."""
    exact = Fraction(x) * Fraction(y) + Fraction(z)
    if exact != 0:
        return float(exact)
    product = math.copysign(0.0, x) * math.copysign(1.0, y)
    return product + z if x * y == 0.0 and z == 0.0 else 0.0   # x y = -z: +0 to nearest


def div_rn_unsigned0(a, b, y):
    q0 = a * y
    q1 = _fma(_fma(-b, q0, a), y, q0)
    return _fma(_fma(-b, q1, a), y, q1)


def _wanted(a, b):
    return 0.0 if a == 0.0 and b > 0.0 else a / b


def test_the_ieee_quotient_but_for_one_zero():
    bad = []
    for a, b in _operands(20000, 0xD1F3):
        q = div_rn_unsigned0(a, b, 1.0 / b)
        if _bits(q) != _bits(_wanted(a, b)):
            bad.append((a, b, q, a / b))
    assert not bad, bad[:5]


def test_zero_dividends():
    for b in (3.0, -3.0, 1.0e-3, -7.5e10):
        for a in (0.0, -0.0):
            q = div_rn_unsigned0(a, b, 1.0 / b)
            assert q == 0.0 and _bits(q) == _bits(_wanted(a, b)), (a, b)
