"""gb_check_single_batch_noalloc while its stream is captured into a graph: batches
that take either form of the single-n kernel, after a first call with another
batch size, replayed on new inputs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 33, 5000, 90_000])
def test_captured_and_replayed(gbmod, oracle, count):
    import torch

    L = gbmod.load()
    f = L.gb_check_single_batch_noalloc
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p,
                                           ctypes.c_uint64, ctypes.c_void_p]
    n = torch.zeros(count, dtype=torch.int64, device="cuda")
    p, q = torch.zeros_like(n), torch.zeros_like(n)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert f(n.data_ptr(), 1, p.data_ptr(), q.data_ptr(), 0, s.cuda_stream) == 0  # the table
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        assert f(n.data_ptr(), count, p.data_ptr(), q.data_ptr(), 0, s.cuda_stream) == 0
    for seed in range(2):
        v = np.random.default_rng([count, seed]).integers(2**20, 2**63, size=count, dtype=np.uint64) * np.uint64(2)
        n.copy_(torch.from_numpy(v.view(np.int64)))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        got = p.cpu().numpy().view(np.uint64)
        np.testing.assert_array_equal(got, oracle.single_minp(v, p_limit=65521))  # GB_NOALLOC_P_LIMIT
        np.testing.assert_array_equal(q.cpu().numpy().view(np.uint64), v - got)
