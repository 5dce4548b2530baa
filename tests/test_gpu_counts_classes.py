"""Partition counts by residue classes, against the oracle: counts of n at
which the modulus changes (2, 6, 30, 210), n from 4 on (where the primes that
divide the modulus are most of the pairs), ragged groups of 32 n, and word
edges of the classes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 31, 33, 97, 200, 481, 1000, 3359, 3361, 7000, 20000])
@pytest.mark.parametrize("start", [4, 6, 10, 190, 2 * 32 * 210 - 64, 65536, 3_000_002])
def test_counts_match_the_sieved_convolution(ctx, start, count):
    top = start + 2 * (count - 1)
    s = np.ones(top + 1, bool)
    s[:2] = False
    for p in range(2, int(top**0.5) + 1):
        if s[p]:
            s[p * p::p] = False
    got = ctx.goldbach_counts(start, count)
    rng = np.random.default_rng(count)
    pick = np.unique(np.concatenate([np.arange(min(count, 40)), np.arange(max(0, count - 40), count),
                                     rng.integers(0, count, size=60)]))
    for j in pick.tolist():
        n = start + 2 * j
        want = int((s[:n // 2 + 1] & s[n - n // 2:n + 1][::-1]).sum())
        assert got[j] == want, n


def test_the_same_n_from_batches_of_all_sizes(ctx):
    start = 10**8 + 2
    big = ctx.goldbach_counts(start, 8000)
    for count in (5, 150, 700):
        np.testing.assert_array_equal(ctx.goldbach_counts(start + 2000, count), big[1000:1000 + count])


@pytest.mark.parametrize("start,count", [(4, 100_003), (190, 131_071), (30_000_000, 1000), (29_999_986, 4096),
                                         (10**7, 2000), (10**7, 480), (10**7, 30), (4_000_000, 1300)])
def test_split_classes_and_single_words(ctx, start, count):
    """Counts that take the classes mod 30 and 210 from the smallest n on, and
    tasks of less than a round of seven words a lane."""
    top = start + 2 * (count - 1)
    s = np.ones(top + 1, bool)
    s[:2] = False
    for p in range(2, int(top**0.5) + 1):
        if s[p]:
            s[p * p::p] = False
    got = ctx.goldbach_counts(start, count)
    rng = np.random.default_rng(count)
    pick = np.unique(np.concatenate([np.arange(12), np.arange(count - 12, count), rng.integers(0, count, size=16)]))
    for j in pick.tolist():
        n = start + 2 * j
        assert got[j] == int((s[:n // 2 + 1] & s[n - n // 2:n + 1][::-1]).sum()), n
