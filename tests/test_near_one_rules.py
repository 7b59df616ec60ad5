"""The rounding rules behind the engine's roots, reciprocals and quotients near
1 and for a known divisor, against exact rational arithmetic: the rule's result
must be the correctly rounded one that sqrt() and '/' give."""
import math
import random
from fractions import Fraction as Fr

import pytest


def down(x):
    """x (near 1) rounded towards minus infinity to a double."""
    u = Fr(1, 2 ** 53) if x < 1 else Fr(1, 2 ** 52)
    return float((x / u).__floor__() * u)


def up(x):
    u = Fr(1, 2 ** 53) if x <= 1 else Fr(1, 2 ** 52)
    return float(-((-x / u).__floor__()) * u)


def near_one_values():
    rng = random.Random(1)
    for m in range(400):
        yield 1 + m * 2.0 ** -52
        yield 1 - m * 2.0 ** -53
    for _ in range(4000):
        yield 1 + rng.randrange(2 ** 25) * 2.0 ** -52
        yield 1 - rng.randrange(2 ** 26) * 2.0 ** -53


def test_root_reciprocal_and_quotient_next_to_one():
    rng = random.Random(2)
    for s in near_one_values():
        if abs(Fr(s) - 1) >= Fr(1, 2 ** 27):
            continue
        length = down(1 + (Fr(s) - 1) / 2)
        assert length == math.sqrt(s)
        inv = up(1 - (Fr(length) - 1))
        assert inv == 1.0 / length
        a = rng.uniform(-1.0, 1.0)
        q = float(Fr(a) - Fr(a) * (Fr(length) - 1))
        r = Fr(a) - Fr(q) * Fr(length)
        assert Fr(float(r)) == r  # the remainder is exact
        assert float(Fr(q) + r * Fr(inv)) == a / length


@pytest.mark.parametrize("divisor", [1.0, 16.0, 128.0, 3.0, 90.50966799187809, 255.99999999999997, 1.0000000000000002,
                                     1.9999999999999998, 0.7071067811865476])
def test_quotient_by_a_known_divisor(divisor):
    rng = random.Random(3)
    y = 1.0 / divisor
    for _ in range(4000):
        a = rng.choice((1.0, -1.0)) * rng.uniform(0.5, 2.0) * 2.0 ** rng.randrange(-40, 20)
        q = a * y
        for _ in range(2):  # the remainder is rounded as an FMA rounds it
            r = float(Fr(a) - Fr(q) * Fr(divisor))
            q = float(Fr(q) + Fr(r) * Fr(y))
        assert q == a / divisor
