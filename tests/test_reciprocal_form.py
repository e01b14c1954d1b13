"""The stage's three-operation division (div_markstein in sac_kernels.cuh) against the
rounded quotient, in exact rational arithmetic, down to the smallest numerators that its
comment allows for each divisor."""
import math
import random
from fractions import Fraction

import pytest


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _form(n, d):
    r = 1.0 / d
    q = n * r
    return _fma(_fma(-q, d, n), r, q)


def _draw(rng, lo, hi):
    return rng.choice((-1, 1)) * math.ldexp(1 + rng.random(), rng.randrange(lo, hi))


@pytest.mark.parametrize("smallest,divisors", [(-807, (-100, 100)), (-960, (-40, 40))])
def test_quotients_down_to_the_smallest_numerators(smallest, divisors):
    rng = random.Random(3)
    for k in range(6000):
        n = _draw(rng, smallest, smallest + 60 if k % 2 else 600)
        d = abs(_draw(rng, *divisors))
        assert _form(n, d) == n / d, (n, d)


def test_a_second_division_by_twelve():
    rng = random.Random(4)
    for k in range(6000):
        n = _draw(rng, -1000, -900 if k % 2 else 600)
        assert _form(n, 12.0) == n / 12.0, n


def test_smaller_numerators_keep_all_but_the_last_bit():
    rng = random.Random(5)
    for _ in range(6000):
        n, d = _draw(rng, -1060, -969), abs(_draw(rng, -100, 100))
        q = n / d
        assert abs(_form(n, d) - q) <= math.ulp(q), (n, d)


def test_zero_numerators():
    for d in (0.3, 12.0, 2.0**-40):
        assert _form(0.0, d) == 0.0 and _form(-0.0, d) == 0.0
