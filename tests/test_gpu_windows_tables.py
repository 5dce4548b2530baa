"""Windows whose q are tested one by one need no sieving primes up to sqrt(top):
far out they run in a context whose tables end below it, beside a window that
is sieved with what it needs itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_far_tested_windows_need_no_far_tables(gbmod, oracle, mode):
    starts = np.array([10**18 + 2, 10**12, 4 * 10**18], dtype=np.uint64)
    counts = np.array([19_000, 50_000, 17_001], dtype=np.uint64)
    n = np.concatenate([np.uint64(s) + np.uint64(2) * np.arange(int(c), dtype=np.uint64)
                        for s, c in zip(starts, counts)])
    want = oracle.single_minp(n, p_limit=10**8).astype(np.uint32)
    with gbmod.Context(0) as c:
        before = c.mem_info()[0]
    with gbmod.Context(0, budget=before + (400 << 20)) as c:  # primes to 2e9 would take 2 GB
        per, minp, s = c.verify_windows(starts, counts, want_minp=True, mode=mode)
        np.testing.assert_array_equal(minp, want)
        assert s["sieved_windows"] == 1 and all(p["failures"] == 0 for p in per)
        with pytest.raises(gbmod.GbError):  # every prime: the tables do not fit
            c.verify_windows(starts, counts, mr_below=1)
