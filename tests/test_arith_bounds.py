"""The bounds that the quotient estimates state, restated in Python: near_inv's
relative error, the large-prime pass's first marks at the smallest primes and
farthest bases that a range's masks use, and n mod M of the single-n sieve for
every modulus it is built with."""
import os
import random
import re
from fractions import Fraction

import numpy as np

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
M32 = (1 << 32) - 1


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def low32(est):
    assert 2.0**52 <= est < 2.0**53
    return int(est) & M32


def near_inv(p):
    r0 = float(np.float32(1.0) / np.float32(p))
    return fma(r0, fma(-float(p), r0, 1.0), r0)


def test_near_inv():
    rng = random.Random(1)
    worst = Fraction(0)
    for i in range(60000):
        e = rng.randrange(14, 32)
        p = (1 << e) + rng.randrange(1 << (e - 1 if i % 2 else 8)) | 1  # just above a power of two: the float's worst
        if p < 1 << 32:
            worst = max(worst, abs(Fraction(near_inv(p)) * p - 1))
    assert Fraction(1, 2**48) < worst <= Fraction(1, 2**46) + Fraction(1, 2**52)


def test_first_marks_of_a_ranges_masks():
    rng = random.Random(2)
    done = 0
    while done < 20000:
        p = rng.choice([(1 << 14) + 27, rng.randrange(1 << 14, 1 << 20) | 1])
        if p % 3 == 0:
            continue
        top = min(p << 42, (1 << 64) // 6)
        g0 = rng.choice([rng.randrange(1 << 30, top), top - 1 - rng.randrange(1 << 12),
                         p * rng.randrange((1 << 30) // p + 1, top // p) + rng.choice([-1, 0, 1, p // 2, p // 6])])
        m = low32(fma(float(g0), near_inv(p), 1.5 * 2.0**52))
        d = (m * p - g0) & M32
        p6 = p // 6
        a1, a5 = (p6, -p6 - 1) if p % 6 == 1 else (-p6 - 1, p6)
        for c, a in ((1, a1), (5, a5)):
            assert min((d + a) & M32, (d + a + p) & M32) == (-c * pow(6, -1, p) - g0) % p, (g0, p, c)
        done += 1


def test_sieve_moduli():
    src = open(os.path.join(ROOT, "goldbach-gpu_b200", "csrc", "kernels", "single.cu")).read()
    mods = [int(v) for v in re.search(r"kMods\[kSieveMods\] = \{(.*?)\}", src, re.S).group(1).replace("\n", "").split(",")]
    prod = [int(np.prod(mods[int(i):int(i) + int(c)])) for i, c in re.findall(r"sieve_group<(\d+), (\d+)>\(tab", src)]
    ones = [int(a) * int(b) * int(c) for a, b, c in re.findall(r"sieve_ones<(\d+), (\d+), (\d+)>\(tab", src)]
    assert len(prod) == 17 and len(ones) == 16
    rng = random.Random(3)
    for m in prod + ones + [(1 << 16) + 1]:
        assert 1 << 16 < m < 1 << 31
        for _ in range(400):
            n = rng.choice([rng.randrange(1 << 64), (1 << 64) - 1 - rng.randrange(1 << 12),
                            min((1 << 64) - 1, max(0, m * rng.randrange((1 << 64) // m) + rng.choice([-1, 0, 1])))])
            est = float(n) * (Fraction(1.0 / m)) + Fraction(3 * 2**51)
            r = (n - low32(float(est)) * m) & M32
            assert min(r, (r + m) & M32) == n % m, (n, m)
