"""Ranges whose chunk width is left open (any multiple of 512 n that fills the
GPU evenly) against the same range cut into chunks of a given power of two, and
per-n output against the oracle where every chunk boundary falls inside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start,count,seg", [
    (4, 2_000_003, 10**7), (4, 5_000_000, 777_777), (10**9, 30_000_001, 10**7), (10**9 - 2, 61_234_567, 2**26),
    (10**12, 150_000_011, 10**7), (10**12 + 2, 45_000_000, 1 << 22), (10**15, 40_000_001, 10**7),
    (10**15 + 4, 300_000_007, 10**8), (10**12, 600_000_000, 10**7),
])
@pytest.mark.parametrize("shards", [1, 3])
def test_open_width_agrees_with_a_given_one(ctx, start, count, seg, shards):
    last = start + 2 * (count - 1)
    kw = dict(seg_size=seg, want_seg=True, shard_index=shards - 1, shard_count=shards)
    r = ctx.verify_range(start, last, **kw)
    g = ctx.verify_range(start, last, chunk=1 << 18, **kw)
    for key in ("checked", "verified", "failures", "max_minp", "phase2_fallbacks", "num_segments"):
        assert r.result[key] == g.result[key], key
    assert r.result["failures"] == 0 and (shards > 1 or r.result["checked"] == count)
    np.testing.assert_array_equal(r.hist, g.hist)
    np.testing.assert_array_equal(r.seg_fallbacks, g.seg_fallbacks)


@pytest.mark.parametrize("start,count", [(4, 1_300_001), (10**9, 3_000_017), (10**12 + 2, 1_000_003)])
def test_open_width_per_n(ctx, oracle, start, count):
    n = np.uint64(start) + np.uint64(2) * np.arange(count, dtype=np.uint64)
    r = ctx.verify_range(start, start + 2 * (count - 1), want_minp=True)
    np.testing.assert_array_equal(r.min_p, oracle.single_minp(n, p_limit=10**8).astype(np.uint32))
