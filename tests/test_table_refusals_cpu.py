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


def demotable(B=1, Hkv=2, nb=4):
    """A table of raw blocks whose demotions stop before the launch, with the rungs they chose."""
    c = PagedLayerCache(PagedPool(10 * 1474560, 128, 32, device="cpu"), B, Hkv, cap_blocks=nb)
    c.offs_h[:], c.level_h[:], c.len_h[:] = c.pool.alloc(16, c.rows * nb).reshape(c.rows, nb), 16, nb * P

    class Planned(Exception):
        pass

    class Lib:
        def __getattr__(self, name):
            return getattr(c.pool.lib, name)

        def gkv_table_demotions(self, offs, level, B, Hkv, cap, blocks, tgt, nb):
            import ctypes
            raise Planned(np.clip(np.array((ctypes.c_int32 * (B * Hkv * nb)).from_address(tgt)), 0, 4).tolist())

    c.lib = Lib()
    return c, Planned


@pytest.mark.parametrize("tgt,error", [(np.zeros((2, 5), np.int32), ValueError), (np.zeros((3, 4), np.int32), ValueError),
                                       (np.full((2, 4), 1.9), IndexError), (np.zeros((2, 4), complex), IndexError)])
def test_targets_that_no_table_of_ladder_indices_can_be_are_refused(tgt, error):
    c, _ = demotable()
    with pytest.raises(error):
        c.apply_demotion(tgt)


@pytest.mark.parametrize("dtype,big", [(np.int64, 1 << 32), (np.uint32, (1 << 32) - 1), (np.int32, 1 << 30), (np.uint8, 255), (np.int64, -(1 << 33))])
def test_targets_of_every_integer_type_count_as_the_nearest_rung(dtype, big):
    c, planned = demotable()
    tgt = np.array([[0, 1, 4, big]] * 2).astype(dtype)
    with pytest.raises(planned) as e:
        c.apply_demotion(tgt)
    assert e.value.args[0] == [0, 1, 4, 0 if big < 0 else 4] * 2


def test_slots_are_asked_for_by_whole_numbers_of_a_rung_on_the_ladder():
    pool = PagedPool(2 * 1474560, 128, 32, device="cpu")
    with pytest.raises(TypeError):
        pool.alloc(16, 2.5)
    with pytest.raises(KeyError):
        pool.alloc(3, 1)
    with pytest.raises(ValueError):
        pool.free(3, pool.alloc(16, 1))
    assert pool.alloc(3, 0).size == 0 and pool.alloc(np.int32(8), np.int64(3)).size == 3
