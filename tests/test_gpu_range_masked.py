"""Ranges through the large-prime masks (short ranges, and ranges far out),
against the oracle: offsets from just above 2^33 to the top of the 64-bit
range, ranges of one chunk and of several segments, ragged segments, shards,
per-n output, given chunk widths and halos, and the same range with and
without the masks (a shard of a wide range takes wide chunks)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expect(oracle, start, count):
    n = np.uint64(start) + np.uint64(2) * np.arange(count, dtype=np.uint64)
    return oracle.single_minp(n, p_limit=10**8).astype(np.uint32)


@pytest.mark.parametrize("start", [8 * 2**30, 8 * 2**30 - 2000, 10**12 - 10**5, 10**15 + 6, 10**18,
                                   2**62 - 4000, 2**64 - 2 - 2 * 8999])
@pytest.mark.parametrize("opts", [dict(seg_size=10**7), dict(seg_size=1000), dict(seg_size=2500, chunk=8192, halo=256)])
def test_per_n_and_segments(ctx, oracle, start, opts):
    count = 9000
    want = expect(oracle, start, count)
    r = ctx.verify_range(start, start + 2 * (count - 1), want_minp=True, want_bits=True, want_seg=True,
                         want_seg_hist=True, p_small=500, **opts)
    np.testing.assert_array_equal(r.min_p, want)
    assert r.result["checked"] == r.result["verified"] == count and r.result["failures"] == 0
    assert r.result["max_minp"] == want.max() and r.result["phase2_fallbacks"] == (want > 500).sum()
    primes = ctx.primes_upto(1 << 16)
    k = np.searchsorted(primes, want)
    for i in range(r.result["num_segments"]):
        part = slice(i * opts["seg_size"], (i + 1) * opts["seg_size"])
        np.testing.assert_array_equal(r.seg_hist[i], np.bincount(np.minimum(k[part], 4095), minlength=4096))
        assert r.seg_fallbacks[i] == (want[part] > 500).sum()
    np.testing.assert_array_equal(r.hist, r.seg_hist.sum(axis=0))
    bits = np.unpackbits(r.verified_bits.view(np.uint8), bitorder="little")
    assert bits[:count].all() and not bits[count:].any()


@pytest.mark.parametrize("start", [10**12 + 2, 10**16])
def test_shards_sum_to_the_whole(ctx, start):
    count = 3_000_017
    kw = dict(seg_size=400_000, want_seg=True)
    whole = ctx.verify_range(start, start + 2 * (count - 1), **kw)
    parts = [ctx.verify_range(start, start + 2 * (count - 1), shard_index=i, shard_count=3, **kw) for i in range(3)]
    np.testing.assert_array_equal(sum(p.hist for p in parts), whole.hist)
    assert sum(p.result["checked"] for p in parts) == count
    assert max(p.result["max_minp"] for p in parts) == whole.result["max_minp"]


def test_failures_within_the_bound(ctx, oracle):
    start, count = 10**15, 20_000
    want = expect(oracle, start, count)
    r = ctx.verify_range(start, start + 2 * (count - 1), p_small=3, phase2_limit=47, want_minp=True, want_bits=True)
    np.testing.assert_array_equal(r.min_p, np.where(want <= 47, want, 0))
    bad = np.nonzero(want > 47)[0]
    assert r.result["failures"] == len(bad) and r.result["first_failure_n"] == start + 2 * int(bad[0])


def test_wide_masked_range_agrees_with_windows(ctx):
    """Several runs of segments (2^28 n each) against the windows pipeline."""
    start, count = 10**15 + 2, (1 << 28) + 12345
    r = ctx.verify_range(start, start + 2 * (count - 1), seg_size=1 << 27)
    per, _, _ = ctx.verify_windows([start], [count], mr_below=1)
    primes = ctx.primes_upto(1 << 20)[:4096].astype(np.uint64)
    assert r.result["verified"] == per[0]["verified"] == count
    assert r.result["max_minp"] == per[0]["max_minp"]
    assert int((r.hist * primes).sum()) == per[0]["minp_sum"]


def test_without_room_for_the_masks(gbmod):
    """A budget that holds the chunks' lists (157 MB) but not the masks (22 MB)
    beside them: the chunks sieve every prime, with the same results."""
    start, count = 10**15 + 2, 1 << 28
    with gbmod.Context(0) as c:
        room = c.mem_info()[0] + (163 << 20)
        want = c.verify_range(start, start + 2 * (count - 1), chunk=1 << 20)
    with gbmod.Context(0, budget=room) as c:
        got = c.verify_range(start, start + 2 * (count - 1), chunk=1 << 20)
    np.testing.assert_array_equal(got.hist, want.hist)
    assert got.result["verified"] == want.result["verified"] == count
    assert got.result["kernel_launches"] < want.result["kernel_launches"]
