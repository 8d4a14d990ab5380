"""The branch-free quotient of common.cuh (div_by): a y, two corrections by the remainder, each a fused
multiply-add. Here in exact rational arithmetic with one rounding per operation, against the division:
equal bits over random operands, quotients next to a rounding boundary, the gas constants' sizes, and
every d whose reciprocal is hard to round (mantissas near 1 and 2)."""
import random
from fractions import Fraction as Q

import pytest


def _fma(a, b, c):
    return float(Q(a) * Q(b) + Q(c))


def _div_by(a, d, y):
    q = a * y
    q = _fma(_fma(-q, d, a), y, q)
    return _fma(_fma(-q, d, a), y, q)


def _operands(kind, rng):
    m = lambda: 1.0 + rng.getrandbits(52) * 2.0 ** -52
    if kind == "random":
        return m() * 2.0 ** rng.randint(-300, 300), m() * 2.0 ** rng.randint(-300, 300)
    if kind == "boundary":                       # a = d (q + half an ulp), rounded: next to a midpoint
        d, q = m(), m()
        return float(Q(d) * (Q(q) + Q(2) ** -53)), d
    if kind == "mantissa":
        u = 2.0 ** -52 * rng.randint(0, 3)
        return m(), (1.0 + u) if rng.random() < 0.5 else (2.0 - 2.0 ** -52 - 2 * u)
    return -rng.uniform(1e2, 1e4), rng.uniform(5.0, 1500.0)


@pytest.mark.parametrize("kind", ["random", "boundary", "mantissa", "physical"])
def test_the_quotient_is_the_divisions(kind):
    rng = random.Random(17)
    for _ in range(20000):
        a, d = _operands(kind, rng)
        assert _div_by(a, d, 1.0 / d) == a / d, (a.hex(), d.hex())
    assert _div_by(0.0, 3.0, 1.0 / 3.0) == 0.0
