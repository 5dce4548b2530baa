"""The base-2 + Lucas primality proof of the single-n kernels, against the
oracle's 7-base Miller-Rabin scan: every batch size at which the split of a
batch over lanes changes, moduli on both sides of 2^62 (where the residues'
range changes), and n whose first candidate q is a strong pseudoprime to
base 2 without a small factor, so that only the Lucas test rejects it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# strong pseudoprimes to base 2 (to the first 5, 6, 7, 9 and 11 prime bases; Jaeschke
# 1993), and the squares of the two Wieferich primes
SPSP2 = [2152302898747, 3474749660383, 341550071728321, 3825123056546413051, 1093**2, 3511**2]


@pytest.mark.parametrize("count", [1, 31, 592, 593, 8191, 8192, 80001])
@pytest.mark.parametrize("bits", [22, 40, 62, 64])
def test_batch_sizes_and_magnitudes(ctx, oracle, count, bits):
    rng = np.random.default_rng(count * 100 + bits)
    n = rng.integers(2 ** (bits - 2), 2 ** (bits - 1), size=count, dtype=np.uint64) * np.uint64(2)
    p, q, r = ctx.check_single(n)
    want = oracle.single_minp(n)
    np.testing.assert_array_equal(p, want)
    np.testing.assert_array_equal(q, n - p)
    assert r.found == count and r.max_p == want.max()


@pytest.mark.parametrize("count", [6, 600, 9000])
def test_base2_pseudoprimes_are_rejected(ctx, oracle, count):
    n = np.array([s + p for s in SPSP2 for p in (3, 5, 311, 313, 317, 331)] +
                 [2**62 - 2 + 2 * i for i in range(4)], dtype=np.uint64)
    n = np.resize(n, count)
    p, _, _ = ctx.check_single(n)
    np.testing.assert_array_equal(p, oracle.single_minp(n))


@pytest.mark.parametrize("p_limit", [3, 100, 312, 313, 316, 317, 500])
@pytest.mark.parametrize("count", [40, 1000, 9000])
def test_candidate_bound_at_the_sieved_block(ctx, oracle, p_limit, count):
    n = np.uint64(10**18) + np.uint64(2) * np.arange(count, dtype=np.uint64)
    p, q, r = ctx.check_single(n, p_limit=p_limit)
    want = oracle.single_minp(n, p_limit=p_limit)
    np.testing.assert_array_equal(p, want)
    assert r.found == (want > 0).sum() and (q[want == 0] == 0).all()
