"""Operands on which correctly rounded quotients and roots can go wrong."""
import numpy as np

N = 2 ** 53


def denominators(rng):
    """Significands near all ones (an odd distance j from a power of two has its
    reciprocal within j^2 / 2^54 units of a midpoint), near one, and random ones."""
    j = np.concatenate([np.arange(1, 4000), 2 * rng.integers(0, 2 ** 25, 20000) + 1, rng.integers(1, 2 ** 40, 20000)])
    m = np.concatenate([N - j, N // 2 + j, N // 2 + np.arange(4000), rng.integers(N // 2, N, 50000)])
    return m.astype(np.float64) * 2.0 ** -52


def roots():
    """Arguments whose root is next to a midpoint of two neighbours: x 2^k = z^2 - d for an odd
    z of 54 bits, where the root is z - d / 2z in units of half a last place.  d is 1 (mod 8)
    and has four roots modulo 2^k, found bit by bit.  With them powers of two and their
    neighbours, and squares."""
    xs = []
    for d in range(-16000, 16000):
        if d % 8 != 1:
            continue
        r = 1                                         # r^2 = d (mod 2^j), one bit more at a time
        for j in range(3, 56):
            if (r * r - d) >> j & 1:
                r += 1 << (j - 1)
        for k in (54, 55):
            for z in (r, -r, r + (1 << (k - 1)), -r + (1 << (k - 1))):
                z %= 1 << k
                lo, hi = (106, 107) if k == 54 else (107, 108)
                if z < 1 << 54 and 1 << lo <= z * z - d < 1 << hi:
                    assert (z * z - d) % (1 << k) == 0
                    xs.append(float((z * z - d) >> k) * 2.0 ** (k - 54 - 52))
    near = [1.0 + i * 2.0 ** -52 for i in range(200)] + [1.0 - i * 2.0 ** -53 for i in range(200)]
    near += [4.0 * v for v in near] + [2.0 * v for v in near] + [float(i * i) for i in range(1, 3000)]
    return np.array(xs + near)


def quotients(rng):
    """Numerators and denominators with x 2^k = d (mod y) for a small d: the quotient is
    next to a midpoint."""
    xs, ys = [N - 3, N - 3, N - 2], [N - 2, N - 1, N - 1]
    for t in range(1500):
        b = (int(rng.integers(N // 2, N)) | 1, N - 1 - 2 * int(rng.integers(2 ** 20)), N - 1 - 2 * int(rng.integers(2 ** 45)))[t % 3]
        half = pow(2, -1, b)
        for k in (53, 54):
            inv = pow(half, k, b)
            for d in range(-7, 8):
                a = d * inv % b
                a += b * (-(-(N // 2 - a) // b)) if a < N // 2 else 0
                for c in (a, a + b):
                    if N // 2 <= c < N:
                        xs.append(c)
                        ys.append(b)
    return np.array(xs, dtype=np.float64) * 2.0 ** -52, np.array(ys, dtype=np.float64) * 2.0 ** -52


def cases(seed):
    """(operation, x, y, expected): 0 recip_rn(y), 1 sqrt_rn(x), 2 x / y by recip_rn and
    quot_rn, 3 low_quot; signs and exponents over the accepted ranges, their ends among them."""
    rng = np.random.default_rng(seed)
    sign = lambda n: rng.choice([-1.0, 1.0], n)
    d = denominators(rng)
    y = np.concatenate([sign(d.size) * d * 2.0 ** e for e in (-100, -60, 0, 59, 99)])
    yield 0, y, y, 1.0 / y
    x = roots()
    x = np.concatenate([x * 2.0 ** e for e in (-100, 0, 96)])
    yield 1, x, x, np.sqrt(x)
    a, b = quotients(rng)
    for ex, ey in ((0, 0), (-860, 0), (-960, -60), (900 - 1, -60), (-960, 59), (850, 99), (-860, 99)):
        x, y = sign(a.size) * a * 2.0 ** ex, sign(b.size) * b * 2.0 ** ey
        yield 2, x, y, x / y
    a, b = np.tile(a, 3), np.tile(b, 3) * 2.0 ** rng.integers(-100, 99, 3 * b.size)
    x = sign(a.size) * a * 2.0 ** rng.integers(-1000, -861, a.size)
    sub = rng.integers(1, N, a.size).astype(np.float64) * 2.0 ** rng.integers(-1074, -1030, a.size).astype(np.float64)
    for v in (x, sub, sign(a.size) * sub * 2.0 ** -20):
        yield 3, v, b, v / b
