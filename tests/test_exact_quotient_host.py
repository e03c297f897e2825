"""The method of claw2_exact.cuh's quotients on the CPU, in exact integers.

q0 = RN(x r), q = RN(q0 + r (x - y q0)) with r = RN(1/y) must be RN(x/y).  The
cases that could break it have a quotient next to the midpoint of two
neighbouring numbers: x 2^k = d (mod y) for a small d, built here with modular
inverses, the largest significands (where r is least accurate) among them; and
the three pairs that the error bound leaves open.
"""
import random
from fractions import Fraction


def _rn(f):
    return f.numerator / f.denominator if f else 0.0       # int / int rounds correctly


def _fma(a, b, c):
    return _rn(Fraction(a) * Fraction(b) + Fraction(c))


def _quot(x, y):
    r = _rn(1 / Fraction(y))
    q = x * r
    return _fma(_fma(-y, q, x), r, q)


def test_quotients_next_to_midpoints():
    n = 2 ** 53
    pairs = [(n - 3, n - 2), (n - 3, n - 1), (n - 2, n - 1)]
    rng = random.Random(1)
    for t in range(1500):
        b = (rng.randrange(n // 2, n) | 1, n - 1 - 2 * rng.randrange(2 ** 20), n - 1 - 2 * rng.randrange(2 ** 45))[t % 3]
        half = pow(2, -1, b)
        for k in (53, 54):
            inv = pow(half, k, b)
            for d in range(-7, 8):
                a = d * inv % b
                a += b * (-(-(n // 2 - a) // b)) if a < n // 2 else 0
                pairs += [(c, b) for c in (a, a + b) if n // 2 <= c < n]
    assert len(pairs) > 20000
    for a, b in pairs:
        x, y = a * 2.0 ** -52, b * 2.0 ** -52
        assert _quot(x, y) == x / y, (a, b)
