"""What moving a few slots costs, natively, where Python's memory tracing does not look."""
import time

import numpy as np
import pytest

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


def test_every_slot_of_a_long_pool_counts_for_its_slab():
    """First and last slots of 110,000 slabs: offsets on and just below the multiples of the slab's bytes."""
    pool = PagedPool(110_000 * 1474560, 128, 32, device="meta")
    offs = pool.alloc(16, 110_000 * 45)
    assert (pool._slab_live == 45).all()
    edge = offs.reshape(110_000, 45)[:, [0, -1]]
    assert (edge % pool.slab_bytes == [0, pool.slab_bytes - 32768]).all()
    pool.free(16, edge.ravel())
    assert (pool._slab_live == 43).all() and pool.slots_in_use(16) == 110_000 * 43


def test_offsets_outside_the_pool_are_refused():
    pool = PagedPool(2 * 1474560, 128, 32, device="meta")
    pool.alloc(16, 90)
    for off in (2 * 1474560, 2 ** 63 - 1, -1, -2 ** 63):
        with pytest.raises(ValueError):
            pool.free(16, np.array([off]))
