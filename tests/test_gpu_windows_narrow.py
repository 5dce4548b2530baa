"""Narrow windows: n by n, tested or sieved, by what the batch costs, with the
same results.  Each form is compared with the pipeline that sieves every window
(mr_below = 1), which the oracle's tests pin down: offsets from 4 to the top of
the 64-bit range and around 2^21 and 2^40, where the paths change, widths at the
rule's lines, both modes, per-n output, bounds that many n fail, and batches on
both sides of the rule's totals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OFFSETS = [4, 6, 2**21 - 300, 2**21, 10**9, 2**40 - 400, 2**40, 10**15, 4 * 10**18]


@pytest.fixture(scope="module")
def far(gbmod):
    with gbmod.Context(0, max_n=2**64 - 2) as c:
        yield c


def both(c, starts, counts, **opts):
    starts, counts = np.array(starts, dtype=np.uint64), np.array(counts, dtype=np.uint64)
    a, ma, sa = c.verify_windows(starts, counts, want_minp=True, **opts)
    b, mb, sb = c.verify_windows(starts, counts, want_minp=True, mr_below=1, **opts)
    np.testing.assert_array_equal(ma, mb)
    assert a == b and (sa["total_n"], sa["failures"]) == (sb["total_n"], sb["failures"])
    assert c.verify_windows(starts, counts, **opts)[0] == a
    return sa["sieved_windows"]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("limit", [0, 1, 2, 3, 5, 47, 9000])
def test_offsets_and_bounds(far, mode, limit):
    for counts in ([1] * 9, [64] * 9, [255] * 9, [256] * 9):
        both(far, OFFSETS, counts, mode=mode, phase2_limit=limit)


@pytest.mark.parametrize("counts", [[255], [256], [16384], [16385], [16384] * 4, [16384] * 5, [300] * 40])
def test_widths_and_totals_of_tested_windows(far, counts):
    starts = 10**18 + 10**6 * np.arange(len(counts))
    assert both(far, starts, counts) == 0


def test_top_of_the_range(far):
    for counts in ([1, 64, 255], [1, 64, 700, 20000]):  # the second batch is tested
        both(far, [2**64 - 2 * c for c in counts], counts)


@pytest.mark.parametrize("narrow", [200, 700])
def test_narrow_windows_beside_a_wide_one(far, narrow):
    """What the narrow windows save is worth a path of its own, or not; those
    below 2^40 are sieved where it is not."""
    starts = [10**12 + 10**5] + [10**11 + 1000 * i for i in range(narrow)] + [10**17 + 1000 * i for i in range(narrow)]
    counts = [30_000] + [5 + i % 90 for i in range(2 * narrow)]
    assert both(far, starts, counts) == (1 if narrow == 700 else 1 + narrow)


def test_options_the_pipeline_refuses(gbmod, far):
    for bad in (dict(halo=100), dict(chunk=1000), dict(block_threads=128), dict(gpu_share_pct=101)):
        for starts, counts in (([10**9], [10]), ([10**18], [100])):
            with pytest.raises(gbmod.GbError):
                far.verify_windows(starts, counts, **bad)


def test_without_room_for_the_n(gbmod):
    """40000 windows of 250 n take 240 MB n by n, and 20 MB of masks."""
    starts, counts = 10**17 + 10**6 * np.arange(40_000, dtype=np.uint64), np.full(40_000, 250, dtype=np.uint64)
    with gbmod.Context(0) as c:
        want = c.verify_windows(starts, counts)[0]
    with gbmod.Context(0) as c:
        c.verify_windows(starts[:4], counts[:4] * np.uint64(100))  # the survivor lists
        room = c.mem_info()[0] + (200 << 20)
    with gbmod.Context(0, budget=room) as c:
        assert c.verify_windows(starts, counts)[0] == want
        assert c.mem_info()[0] <= room
