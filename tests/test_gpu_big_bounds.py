"""gb_check_big with a bound that leaves no candidate: its figures are this
call's, whatever an earlier call left in the context's staging buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", ["nothing", "range", "single", "big"])
@pytest.mark.parametrize("p_limit", [1, 2])
def test_no_candidate_below_the_bound(gbmod, before, p_limit):
    with gbmod.Context(0) as c:
        if before == "range":
            c.verify_range(10**10, 10**10 + 2 * (10**6 - 1))
        elif before == "single":
            c.check_single(np.arange(10**12, 10**12 + 200_000, 2, dtype=np.uint64))
        elif before == "big":
            c.check_big(2**100 + 2)
        p, q, r = c.check_big(2**100, p_limit=p_limit)
        assert (p, q) == (0, 0)
        assert r["candidates"] == 0 and r["mr_tests"] == 0
