"""The branch-free quotient (div_pos.cuh) over the rest of its domain, and the quotients
derived from it in k_cea.cu, in exact arithmetic as in test_division.py: negative
denominators (LU pivots), denominators down to 1e-300, x times the reciprocal of a pivot
with one remainder correction, and x over a small whole number."""
from fractions import Fraction as Fr

import numpy as np
import pytest

from test_division import div_pos, rnd, ulp


def seed_of(b, rng, p):
    """an approximate reciprocal up to 2^-21 off"""
    return rnd((1 / b) * (1 + Fr(float(rng.uniform(-1, 1))) * Fr(1, 2 ** 21)), p)


def test_denominators_of_either_sign_and_of_any_size():
    p, rng = 53, np.random.default_rng(6)
    for k in range(2000):
        b = Fr(float(rng.choice([-1, 1]) * 10.0 ** rng.uniform(-30, 30)))
        if k % 4 == 0:
            b = Fr(1e-300) * (1 if k % 8 else Fr(float(rng.uniform(1, 1e3))))
        a = Fr(1) if k % 3 == 0 else Fr(float(rng.choice([-1, 1]) * 10.0 ** rng.uniform(-8, 7)))
        y0 = seed_of(b, rng, p)
        q = div_pos(a, b, y0, p)
        assert abs(q - a / b) <= ulp(a / b, p), (float(a), float(b))
        assert div_pos(a, -b, -y0, p) == -q


def test_quotient_by_a_pivots_reciprocal():
    p, rng = 53, np.random.default_rng(7)
    fma = lambda x, y, z: rnd(x * y + z, p)
    for _ in range(2000):
        a = Fr(float(rng.choice([-1, 1]) * 10.0 ** rng.uniform(-30, 8)))
        x = Fr(float(rng.choice([-1, 1]) * 10.0 ** rng.uniform(-20, 20)))
        y = div_pos(Fr(1), a, seed_of(a, rng, p), p)
        q = rnd(x * y, p)
        assert abs(fma(fma(-a, q, x), y, q) - x / a) <= ulp(x / a, p)


@pytest.mark.parametrize("d", [3, 5, 6, 12, 20])
def test_quotient_by_a_small_whole_number(d):
    """Correctly rounded: the powers of T keep the bits of a division."""
    p, rng = 53, np.random.default_rng(d)
    fma = lambda x, y, z: rnd(x * y + z, p)
    r = rnd(Fr(1, d), p)
    for _ in range(2000):
        x = Fr(float(rng.choice([-1, 1]) * 10.0 ** rng.uniform(-12, 20)))
        q = rnd(x * r, p)
        assert fma(fma(Fr(-d), q, x), r, q) == rnd(x / d, p)
