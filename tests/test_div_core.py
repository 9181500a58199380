"""The division of the warp-per-cell restarts (div_core in
opencaeporo_b200/csrc/flash_div.cuh) replayed in exact rational arithmetic:
from a reciprocal approximation of relative error up to 2^-19, the refined
and corrected quotient equals Python's correctly rounded a / b, on random
mantissas, divisors next to a power of two, and the hardest cases (quotients
as near the middle of two numbers as two 53-bit operands allow). Divisors
whose mantissa is all ones are the kernel's to hand to the `/` operator; the
test shows that they have to be."""
import random
from fractions import Fraction as F

import pytest


def _rn(x):
    return F(float(x))  # CPython rounds a Fraction correctly


def _fma(a, b, c):
    return _rn(a * b + c)


def _core(a, b, y0):
    e = _fma(-b, y0, F(1))
    t = _fma(e, e, e)
    y1 = _fma(y0, t, y0)
    q1 = _fma(_rn(a * y0), t, _rn(a * y0))
    y = _fma(y1, _fma(-b, y1, F(1)), y1)
    q2 = _fma(_fma(-b, q1, a), y1, q1)
    return _fma(_fma(-b, q2, a), y, q2)


def _operands(kind, rng):
    a, b = (1 << 52) | rng.getrandbits(52), (1 << 52) | rng.getrandbits(52)
    if kind == "near two":
        b = (1 << 53) - 2 - rng.randrange(8)
    elif kind == "near one":
        b = (1 << 52) + rng.randrange(8)
        a = (1 << 52) + rng.randrange(8)
    elif kind == "hard":
        # a 2^54 = m b -+ 1: a / b one part in b 2^54 from a 54-bit number
        b |= 1
        s = rng.choice((1, -1))
        m = (pow(b, -1, 1 << 54) * s) % (1 << 54)
        a = max(1, (m * b - s) >> 54)
        while a < 1 << 52:
            a <<= 1
    return a, b


@pytest.mark.parametrize("kind", ["random", "near two", "near one", "hard"])
def test_div_core_is_correctly_rounded(kind):
    rng = random.Random(kind)
    for _ in range(4000):
        ia, ib = _operands(kind, rng)
        if ib == (1 << 53) - 1:
            continue
        a, b = F(ia), F(ib)
        y0 = _rn(1 / b * (1 + F(rng.randrange(-(1 << 20), 1 << 20), 1 << 39)))
        assert _core(a, b, y0) == _rn(a / b), (ia, ib)


def test_all_ones_divisor_needs_the_general_division():
    b = F((1 << 53) - 1)
    a = F(1 << 52)
    assert _core(a, b, _rn(1 / b * (1 - F(1, 1 << 20)))) != _rn(a / b)
