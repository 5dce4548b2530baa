"""A server started after a large call, under a budget that does not hold both:
the buffers that the context keeps from the call make room for the server's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POOL = 512 << 20


def serve(c, reqs):
    c.serve_start(pool_bytes=POOL)
    held = c.mem_info()[0]
    got = [c.wait(t, 60000) for t in c.submit(*zip(*reqs))]
    c.serve_stop()
    return held, [(g["status"], g["verified"], g["max_minp"], g["minp_sum"]) for g in got]


def test_kept_buffers_make_room_for_the_server(gbmod):
    n = np.arange(10**12, 10**12 + 2 * 16_000_000, 2, dtype=np.uint64)  # 384 MB of n, p and q
    reqs = [(1, 10**15, 100_000), (0, 10**18, 1), (1, 10**12, 50)]
    with gbmod.Context(0, max_n=2**64 - 2) as c:
        held, want = serve(c, reqs)
    assert all(w[0] == 0 for w in want)
    with gbmod.Context(0, max_n=2**64 - 2, budget=held + (64 << 20)) as c:
        p = c.check_single(n)[0]
        assert (p > 0).all()
        got = serve(c, reqs)[1]
        np.testing.assert_array_equal(c.check_single(n)[0], p)
        assert c.mem_info()[0] <= c.mem_info()[1]
    assert got == want
