"""What moving a few slots costs, natively, where Python's memory tracing does not look."""
import time

import numpy as np

from geodesia_kv_b200.paged import PagedPool


def test_moving_a_few_slots_takes_no_longer_in_a_long_pool():
    """Some slabs empty at every step.  A pass over the 880 KB of per-slab arrays of a pool of 160 GB takes 20 us and more, the
    steps themselves 2 to 10; the quickest of many rounds is compared, with a factor of 3."""
    def seconds(slabs):
        pool = PagedPool(slabs * 1474560, 128, 32, device="meta")
        pool.alloc(16, 500)
        best = np.inf
        for _ in range(30):
            t = time.perf_counter()
            for _ in range(20):
                pool.free(16, pool.alloc(16, 100))
            best = min(best, time.perf_counter() - t)
        return best / 20
    short, long = seconds(500), seconds(110_000)
    assert long < 3 * short + 5e-6, (short, long)
