"""Quotient estimates of the far windows, restated in Python and checked on the
CPU:

* the chunk sieve's G0 mod p beyond 2^53 (near_mod, kernels/sieve6.cuh), for
  G0 < 2^61 and 2^14 < p < 2^31;
* the large-prime pass's first marks (win_large_kernel, kernels/windows.cu):
  for every p > 2^20 below 2^32 and mask below 2^27 bits, t_c is (a_c - g0) mod
  p whenever that lies in the mask, and beyond the mask otherwise.
"""
import random
from fractions import Fraction

import numpy as np
import pytest

M32 = (1 << 32) - 1


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def low32(est):
    assert 2.0**52 <= est < 2.0**53
    return int(est) & M32


def test_sieve_remainder_of_far_windows():
    rng = random.Random(3)
    for _ in range(20000):
        p = rng.choice([16411, (1 << 31) - 1, rng.randrange(1 << 14, 1 << 21) | 1, rng.randrange(1 << 14, 1 << 31) | 1])
        g0 = rng.choice([(1 << 61) - 1 - rng.randrange(1 << 12), rng.randrange(1 << 53, 1 << 61),
                         rng.randrange(1, (1 << 61) // p) * p + rng.choice([-1, 0, 1])])
        g0 = min(g0, (1 << 61) - 1)
        magic = ((1 << 64) - 1) // p
        est = fma(float(g0) * 2.0**-64, float(magic), 1.5 * 2.0**52)
        r = (g0 - low32(est) * p) & M32
        assert min(r, (r + p) & M32) == g0 % p, (g0, p)


def first_marks(g0, p):
    pd = float(p)
    r0 = float(np.float32(1.0) / np.float32(p))  # __frcp_rn((float)p)
    inv = fma(r0, fma(-pd, r0, 1.0), r0)
    m = low32(fma(float(g0), inv, 1.5 * 2.0**52))
    d = (m * p - g0) & M32
    p6 = p // 6
    a1, a5 = (p6, -p6 - 1) if p % 6 == 1 else (-p6 - 1, p6)
    padd = p if p < 1 << 31 else 0
    return [min((d + a) & M32, (d + a + padd) & M32) for a in (a1, a5)]


@pytest.mark.parametrize("lo,hi", [((1 << 20) + 1, 1 << 22), (1 << 28, 1 << 31), (1 << 31, 1 << 32)])
def test_large_pass_first_marks(lo, hi):
    rng = random.Random(lo)
    done = 0
    while done < 20000:
        p = rng.choice([lo | 1, rng.randrange(lo, hi) | 1])
        if p % 3 == 0:
            continue
        g0 = rng.choice([rng.randrange(1 << 30, (1 << 64) // 6), (1 << 64) // 6 - rng.randrange(1 << 20),
                         p * rng.randrange(1 << 12, (1 << 64) // 6 // p) + rng.choice([-1, 0, 1, p // 2, p // 6])])
        lbits = rng.choice([32, 1 << 20, (1 << 27) - 32])
        for c, got in zip((1, 5), first_marks(g0, p)):
            want = (-c * pow(6, -1, p) - g0) % p  # 6 (g0 + t) + c = 0 (mod p)
            if want < lbits:
                assert got == want, (g0, p, c)
            else:
                assert got >= lbits, (g0, p, c)
        done += 1
