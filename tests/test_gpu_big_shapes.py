"""gb_check_big at the edges of its lane shapes (8, 16 and 32 lanes of one limb,
then 2, 3, 4 and 5 limbs a lane), against the big-n oracle: bit lengths where
the limbs of R change, n just above a power of two (where q's bit length
depends on p), primes plus 3, 5 and 7 at the widest shapes, and composites
that pass base 2."""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
# the largest prime below 2^bits is 2^bits - c
BELOW = {2047: 85, 2048: 1557, 3071: 187, 3072: 47, 4095: 1615, 4096: 2549}


@pytest.fixture(scope="module")
def B():
    spec = importlib.util.spec_from_file_location("big_oracle", os.path.join(ROOT, "oracle", "big_oracle.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    mod.PR = mod.small_primes(10**6)
    return mod


@pytest.mark.parametrize("bits", [65, 94, 95, 96, 97, 253, 254, 255, 256, 257, 509, 510, 511, 512, 513, 1021, 1022,
                                  1023, 1024, 1025])
def test_bit_lengths_at_the_shapes_edges(ctx, B, bits):
    rng = np.random.default_rng(bits)
    x = sum(int(v) << (32 * i) for i, v in enumerate(rng.integers(0, 2**32, size=bits // 32 + 1, dtype=np.uint64)))
    n = (x & ((1 << bits) - 1) | 1 << (bits - 1)) & ~1
    p, q, _ = ctx.check_big(n)
    assert p == B.minimal_p(n, primes=B.PR) and q == n - p


@pytest.mark.parametrize("k", [65, 96, 254, 255, 256, 510, 512])
@pytest.mark.parametrize("d", [0, 2, 50, 400])
def test_just_above_a_power_of_two(ctx, B, k, d):
    n = 2**k + d
    p, q, _ = ctx.check_big(n)
    assert p == B.minimal_p(n, primes=B.PR) and q == n - p


@pytest.mark.parametrize("bits", list(BELOW))
def test_widest_shapes_prove_a_prime(ctx, B, bits):
    q0 = 2**bits - BELOW[bits]
    p, q, _ = ctx.check_big(q0 + 3, p_limit=50)
    assert (p, q) == (3, q0)
    want = B.minimal_p(q0 + 7, p_limit=7, primes=B.PR)
    assert ctx.check_big(q0 + 7, p_limit=7)[0] == want


@pytest.mark.parametrize("p", [3, 5, 11])
def test_base2_pseudoprime_beyond_64_bits(ctx, B, p):
    """n - p a strong pseudoprime to base 2 (and to every prime base up to 31;
    Arnault 1995's first example exceeds 64 bits): another base rejects it."""
    s = 1195068768795265792518361315725116351898245581
    assert B.sprp(s, 2) and not B.is_probable_prime(s)
    got, q, _ = ctx.check_big(s + p)
    assert got == B.minimal_p(s + p, primes=B.PR) and q == s + p - got


@pytest.mark.parametrize("bits,d", [(200, 798), (256, 908), (400, 196), (512, 660)])
def test_minimal_p_beyond_the_first_batch(ctx, B, bits, d):
    """Every candidate of the first batch (two for each bit of n, at least 512) fails."""
    n = 2 ** (bits - 1) + d
    p, q, r = ctx.check_big(n)
    assert p == B.minimal_p(n, primes=B.PR) and q == n - p
    assert p > B.PR[max(512, 2 * bits)] and r["candidates"] > max(512, 2 * bits)


@pytest.mark.parametrize("bits,d,p", [(96, 1778, 2333), (96, 45472, 691), (250, 774, 3217), (250, 1452, 2473),
                                      (512, 356, 2357), (512, 492, 1753)])
def test_first_prime_at_the_end_of_the_spread_bases(ctx, B, bits, d, p):
    """The first prime n - p is the 32nd or the 33rd candidate without a factor
    below 4096: the other bases run beside base 2 on 32 of them."""
    n = 2 ** (bits - 1) + d
    assert B.minimal_p(n, primes=B.PR) == p
    assert ctx.check_big(n)[:2] == (p, n - p)
