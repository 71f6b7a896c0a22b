"""What the block pool and its tables refuse, they leave as it was."""
import numpy as np
import pytest

from geodesia_kv_b200.paged import LADDER, PagedLayerCache, PagedPool, PoolExhausted, _addr

P = 64


def state(pool):
    return [s.tolist() for s in pool._stack.values()] + [pool._free_slabs, pool._slab_rung.tolist(), pool._slab_live.tolist(), pool._counters.tolist()]


@pytest.mark.parametrize("wrong", [0, 1, 2, 3])
def test_a_release_or_a_demotion_that_is_refused_changes_nothing(wrong):
    """An offset of another rung among those that go back: nothing goes back, so a second call cannot give a slot back twice."""
    pool = PagedPool(10 * 1474560, 128, 32, device="cpu")
    c = PagedLayerCache(pool, 1, 2, cap_blocks=4)
    levels = np.array([[16, 8, 4, 2], [16, 16, 8, 1]], dtype=np.int32)
    for lv in LADDER:
        c.offs_h[levels == lv] = pool.alloc(lv, int((levels == lv).sum()))
    c.level_h[:] = levels
    good = c.offs_h[1, wrong]
    c.offs_h[1, wrong] = pool.alloc(LADDER[(LADDER.index(levels[1, wrong]) + 2) % 5], 1)[0]
    before, offs = state(pool), c.offs_h.copy()
    assert c.lib.gkv_table_release(pool.handle, _addr(c.offs_h), _addr(c.level_h), 8) != 0
    assert state(pool) == before and (c.offs_h == offs).all() and (c.level_h == levels).all()
    flat = np.arange(8)
    lo, ln = levels.ravel().copy(), np.ones(8, np.int32)
    assert c.lib.gkv_table_apply_demotion(pool.handle, _addr(c.offs_h), _addr(c.level_h), 8, *map(_addr, (offs.ravel(), offs.ravel(), flat, lo, ln))) != 0
    assert state(pool) == before and (c.offs_h == offs).all() and (c.level_h == levels).all()
    c.offs_h[1, wrong] = good
    assert c.lib.gkv_table_release(pool.handle, _addr(c.offs_h), _addr(c.level_h), 8) == 0
    assert pool.bytes_in_use == pool.slot[LADDER[(LADDER.index(levels[1, wrong]) + 2) % 5]] and (c.level_h == 0).all()


def test_a_demotion_that_does_not_fit_changes_nothing():
    """Slots of 8 bits would fit, slots of 4 bits would not: the former are not taken, so neither the peak nor the order in which
    slots are handed out changes."""
    pool = PagedPool(4 * 1474560, 128, 32, device="cpu")         # four slabs
    eights = pool.alloc(8, 3 * 80)
    c = PagedLayerCache(pool, 1, 1)
    c.offs_h[0, :40], c.level_h[0, :40], c.len_h[0] = pool.alloc(16, 40), 16, 40 * P
    pool.free(8, eights[7:27])
    pool._counters[2] = pool._counters[1]
    before, tgt = state(pool), np.zeros((1, 40), dtype=np.int32)
    tgt[0, 10:20], tgt[0, 20:30] = LADDER.index(8), LADDER.index(4)
    with pytest.raises(PoolExhausted):
        c.apply_demotion(tgt)
    assert state(pool) == before and (c.level_h[0, :40] == 16).all()
