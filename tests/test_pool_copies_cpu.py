"""Copies and pickles of a block pool."""
import copy
import gc
import pickle

import numpy as np
import pytest

from geodesia_kv_b200.paged import LADDER, PagedPool


def used_pool():
    pool = PagedPool(20 * 1474560, 128, 32, device="cpu")
    held = {r: pool.alloc(r, 30 + r) for r in LADDER}
    for r in LADDER:
        pool.free(r, held[r][::3])
    pool.data[:8] = 7
    return pool, held


def books(pool):
    return [s.tolist() for s in pool._stack.values()] + [pool._free_slabs, pool._slab_rung.tolist(), pool._slab_live.tolist(),
                                                         pool.bytes_in_use, pool.peak_bytes_in_use, pool.bytes_reserved]


@pytest.mark.parametrize("copied", [copy.deepcopy, lambda p: pickle.loads(pickle.dumps(p))])
def test_a_deep_copy_goes_on_by_itself(copied):
    pool, held = used_pool()
    other = copied(pool)
    before = books(pool)
    assert books(other) == before and other.data.data_ptr() != pool.data.data_ptr() and (other.data[:8] == 7).all()
    first = {r: pool.alloc(r, 50).tolist() for r in LADDER}
    assert books(other) == before                                   # untouched by what the first one hands out
    assert {r: other.alloc(r, 50).tolist() for r in LADDER} == first and books(other) == books(pool)
    del pool
    gc.collect()
    for r in LADDER:
        other.free(r, np.concatenate([np.array(first[r]), np.delete(held[r], np.s_[::3])]))
    assert other.bytes_in_use == 0 and other.bytes_reserved == 0


def test_a_shallow_copy_shares_the_bookkeeping_for_as_long_as_either_lives():
    pool, _ = used_pool()
    other = copy.copy(pool)
    a = pool.alloc(8, 10)
    assert books(other) == books(pool) and not set(a) & set(other.alloc(8, 10))
    before = books(pool)
    del pool
    gc.collect()
    assert books(other) == before
    other.free(8, a)


def test_the_peak_can_be_set_back():
    pool, held = used_pool()
    assert pool.peak_bytes_in_use > pool.bytes_in_use
    pool.peak_bytes_in_use = pool.bytes_in_use
    pool.alloc(16, 1)
    assert pool.peak_bytes_in_use == pool.bytes_in_use
