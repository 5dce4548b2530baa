"""Several threads, each with a context of its own on the same device, whose
batches need chunks of different widths (and so different amounts of shared
memory for the same kernel): every call succeeds, with the results it has
alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["windows", "range"])
def test_calls_with_different_chunk_widths(gbmod, call):
    def one(c, chunk):
        if call == "windows":
            return c.verify_windows([10**12], [30_000], chunk=chunk, mr_below=1)[0]
        return c.verify_range(10**12, 10**12 + 2 * 29_999, chunk=chunk).hist.tolist()

    widths = [1 << 13, 1 << 20, 1 << 16, 1 << 18]
    with gbmod.Context(0) as c:
        want = one(c, 0)
    errors, barrier = [], threading.Barrier(len(widths))

    def work(chunk):
        try:
            with gbmod.Context(0) as c:
                barrier.wait()
                for _ in range(400):
                    if one(c, chunk) != want:
                        raise AssertionError("another result")
        except Exception as e:
            errors.append((chunk, repr(e)))

    threads = [threading.Thread(target=work, args=(w,)) for w in widths]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
