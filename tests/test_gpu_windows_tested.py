"""Windows whose masks come from a short sieve and primality tests, against
the oracle's single-n search: offsets on both sides of 2^62 and at the top of
the 64-bit range, widths at the edges of a mask word, a run of 32 words, a
presieve tile and a chunk, and batches that mix them with sieved windows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expect(oracle, starts, counts):
    ns = np.concatenate([np.uint64(s) + np.uint64(2) * np.arange(int(c), dtype=np.uint64)
                         for s, c in zip(starts, counts)])
    return oracle.single_minp(ns, p_limit=10**8).astype(np.uint32)


def check(ctx, oracle, starts, counts, **opts):
    per, minp, summ = ctx.verify_windows(starts, counts, want_minp=True, mr_divisor=1, **opts)
    want = expect(oracle, starts, counts)
    np.testing.assert_array_equal(minp, want)
    off = 0
    for i, c in enumerate(int(c) for c in counts):
        w = want[off:off + c]
        assert per[i] == {"verified": c, "failures": 0, "max_minp": int(w.max()),
                          "minp_sum": int(w.astype(np.uint64).sum())}
        off += c
    # without per-n output the chunks are wider
    per2, _, _ = ctx.verify_windows(starts, counts, mr_divisor=1, **opts)
    assert per2 == per
    return summ


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("lo", [2 * 10**12, 10**18, 2**62 - 10**6, 2**64 - 2 - 2 * 10**6])
def test_widths_and_offsets(ctx, oracle, lo, mode):
    counts = np.array([64, 65, 95, 96, 97, 3071, 3072, 3073, 9000, 20011], dtype=np.uint64)
    gaps = np.arange(len(counts), dtype=np.uint64) * np.uint64(44444)
    starts = np.uint64(lo + lo % 2) + gaps
    s = check(ctx, oracle, starts, counts, mode=mode)
    assert s["sieved_windows"] == 0


def test_last_window_ends_at_the_top(ctx, oracle):
    counts = np.array([1, 64, 700], dtype=np.uint64)
    check(ctx, oracle, np.array([2**64 - 2 * int(c) for c in counts], dtype=np.uint64), counts)


@pytest.mark.parametrize("halo", [128, 4096])
def test_small_halo_and_mixed_batch(ctx, oracle, halo):
    """A window below 2^40 (sieved), tested ones, single n; a halo of 128 sends
    many n to the device Phase 2."""
    starts = np.array([1000, 10**18 + 2, 3 * 10**17, 10**16, 10**12 - 10**6], dtype=np.uint64)
    counts = np.array([5000, 3000, 10, 1, 4000], dtype=np.uint64)
    s = check(ctx, oracle, starts, counts, halo=halo)
    assert s["sieved_windows"] == 2


def test_wide_window_agrees_with_the_full_sieve(ctx):
    """Several presieve tiles and chunks: the same figures as sieving by every prime."""
    starts = np.array([5 * 10**17, 10**15 + 4], dtype=np.uint64)
    counts = np.array([3_000_001, 700_000], dtype=np.uint64)
    a, _, sa = ctx.verify_windows(starts, counts, mr_divisor=1)
    b, _, sb = ctx.verify_windows(starts, counts, mr_below=1)
    assert a == b and sa["sieved_windows"] == 0 and sb["sieved_windows"] == 2


def test_kept_buffers_are_given_back(gbmod):
    """A context whose budget the masks of a wide batch nearly fill: later calls
    that need the room get it, and the same results as in a roomy context."""
    starts = np.array([10**13 + 2], dtype=np.uint64)
    counts = np.array([2 * 10**9], dtype=np.uint64)  # 170 MB of masks
    want = None
    for budget in (0, 720 << 20):  # the range call alone holds 684 MB
        with gbmod.Context(0, budget=budget) as c:
            a, _, _ = c.verify_windows(starts, counts)
            r = c.verify_range(10**12, 10**12 + 2 * (10**8 - 1), want_minp=True)  # 400 MB out
            b, _, _ = c.verify_windows(starts, counts)
            got = (a, b, int(r.min_p.astype(np.uint64).sum()))
            held, room = c.mem_info()
            assert held <= room
        want = want or got
        assert got == want and a == b
