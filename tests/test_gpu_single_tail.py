"""Batches whose warps end with candidates still to be proved: each warp hands
what it has pending to its CTA's list after its last round, and other lanes
than those that gathered an entry copy it there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WARPS = 148 * 16  # of a full launch


@pytest.mark.parametrize("count", [33, 16 * 31, WARPS + 1, 3 * WARPS - 1, 33 * WARPS + 17])
def test_pending_at_the_end(ctx, oracle, count):
    for seed in range(3):
        n = np.random.default_rng([count, seed]).integers(2**20, 2**63, size=count, dtype=np.uint64) * np.uint64(2)
        p, q, r = ctx.check_single(n)
        want = oracle.single_minp(n)
        np.testing.assert_array_equal(p, want)
        np.testing.assert_array_equal(q, n - p)
        assert r.found == count and r.max_p == want.max()
