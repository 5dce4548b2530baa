"""What a context keeps from its calls is bounded in all, not only by buffer:
three calls that each leave 720 MB in a slot of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_kept_buffers_are_bounded_in_all(gbmod):
    n0, small, wide = 10**12, 2**17, 180_000_000
    with gbmod.Context(0) as c:

        def calls(singles, count):
            p = c.check_single(np.arange(n0, n0 + 2 * singles, 2, dtype=np.uint64))[0]
            r = c.verify_range(n0, n0 + 2 * (count - 1), want_minp=True, want_bits=True)
            w = c.verify_windows([n0], [count], want_minp=True)[1]
            np.testing.assert_array_equal(r.min_p[:singles], p[:count])
            np.testing.assert_array_equal(w, r.min_p)
            return c.mem_info()[0]

        wide_lists = c.verify_range(10**9, 10**9 + 2 * (10**9 - 1))  # the widest chunks' survivor lists
        assert wide_lists.result["failures"] == 0
        base = calls(small, small)
        assert calls(30_000_000, wide) <= base + (2 << 30)
        calls(small, small)
