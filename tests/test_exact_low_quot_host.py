"""low_quot of claw2_exact.cuh restated with exact FMAs: quotients whose numerator is
below 2^-860, down to subnormal results, are the bits of the IEEE division."""
import random
import struct

from test_exact_quotient_host import _fma, _quot


def _low_quot(x, y):
    xs = x * 2.0 ** 300
    s = _quot(xs, y)
    if 0.0 < abs(s) < 2.0 ** -722:
        e = _fma(-y, s, xs)
        bits = struct.unpack("<q", struct.pack("<d", s))[0]
        if e != 0.0 and ((bits & 1) != 0) == (abs(s) >= 2.0 ** -723):
            bits += 1 if (e > 0.0) == (s > 0.0) else -1
        s = struct.unpack("<d", struct.pack("<q", bits))[0]
    return s * 2.0 ** -300


def test_quotients_down_to_subnormal_ones():
    rng = random.Random(5)
    for k in range(20000):
        y = rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-6, 6)
        e = rng.choice([rng.randint(-1074, -1000), rng.randint(-1030, -1015), rng.randint(-1000, -861)])
        x = rng.choice([-1.0, 1.0]) * (rng.randint(1, 2 ** 53 - 1) * 2.0 ** -53) * 2.0 ** max(e, -1000) * 2.0 ** min(e + 1000, 0)
        if k % 3 == 0:                     # midpoints of the results' grid, and just off them
            q = (2 * rng.randint(0, 2 ** 20) + 1) * 5e-324
            y = rng.choice([2.0, 0.5, 4.0, 1.0 + 2.0 ** -30, 2.0 - 2.0 ** -40])
            x = q * 0.5 * y if rng.random() < 0.5 else q
        assert _low_quot(x, y) == x / y, (x, y)
