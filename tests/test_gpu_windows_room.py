"""A batch whose windows take both paths, under a budget that holds the buffers
of either but not of both: the second path gets the first one's room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_paths_of_one_batch_share_the_budget(gbmod):
    starts = np.array([10**12, 10**13], dtype=np.uint64)
    counts = np.array([34_000_000, 2 * 10**9], dtype=np.uint64)  # 816 MB n by n; 170 MB of masks
    with gbmod.Context(0, max_n=10**14) as c:
        c.verify_windows(starts[:1], [1000], mr_below=1)  # the survivor lists
        room = c.mem_info()[0] + (880 << 20)
        want = c.verify_windows(starts, counts, mr_below=10**8)[0]
    with gbmod.Context(0, max_n=10**14, budget=room) as c:
        assert c.verify_windows(starts, counts, mr_below=10**8)[0] == want
        assert c.mem_info()[0] <= room
