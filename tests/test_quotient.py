"""The quotient of csrc/wg_div.cuh (one multiplication and two FMAs with the rounded reciprocal of the
divisor), restated in exact rational arithmetic with one rounding per operation, is the correctly
rounded quotient bit for bit; and the exponent range it is used in keeps every intermediate normal."""
import random
from fractions import Fraction as F

import pytest


def rn(v):
    return float(v)  # Fraction -> float is correctly rounded


def quotient(a, b):
    z = rn(F(1) / F(b))
    q = rn(F(a) * F(z))
    r = rn(F(a) - F(b) * F(q))
    return rn(F(q) + F(r) * F(z)), (q, r)


@pytest.mark.parametrize("kind", ["random", "divisor near a power of two", "quotient near one", "exact", "ends of the range"])
def test_quotient_is_correctly_rounded(kind):
    rng = random.Random(kind)
    for _ in range(4000):
        a, b = rng.uniform(1, 2), rng.uniform(1, 2)
        if kind == "divisor near a power of two":
            b = 2.0 - rng.randrange(1, 200) * 2.0 ** -52 if rng.random() < 0.5 else 1.0 + rng.randrange(200) * 2.0 ** -52
        elif kind == "quotient near one":
            a = b + rng.randrange(-8, 9) * 2.0 ** -52
        elif kind == "exact":
            a, b = float(rng.randrange(1, 2 ** 26)), float(rng.randrange(1, 2 ** 26))
            a *= b
        elif kind == "ends of the range":
            a *= 2.0 ** rng.choice([-500, -499, 0, 499, 500])
            b *= 2.0 ** rng.choice([-500, 0, 500])
        else:
            a *= 2.0 ** rng.randrange(-60, 60)
            b *= 2.0 ** rng.randrange(-60, 60)
        if rng.random() < 0.5:
            a = -a
        got, (q, r) = quotient(a, b)
        assert got == a / b
        # no intermediate is subnormal or overflows
        assert 2.0 ** -1022 <= abs(q) < 2.0 ** 1023
        assert r == 0 or 2.0 ** -1022 <= abs(r)
