"""Host logic of the paged pool (size-class free lists over slabs); no GPU needed."""
from __future__ import annotations

import numpy as np
import pytest


def make_pool(mib=32, D=128, group=32):
    from geodesia_kv_b200.paged import PagedPool
    return PagedPool(mib << 20, D, group, device="cpu")


def test_slot_sizes_and_slab_geometry():
    pool = make_pool()
    assert pool.slot == {16: 32768, 8: 18432, 4: 10240, 2: 6144, 1: 512}
    assert pool.slab_bytes == 1474560 and all(pool.slab_bytes % s == 0 for s in pool.slot.values())
    small = make_pool(D=64)
    assert small.slot == {16: 16384, 8: 9216, 4: 5120, 2: 3072, 1: 256}


def test_slots_are_disjoint_and_aligned():
    pool = make_pool()
    got = []
    for rung, n in ((16, 50), (8, 90), (4, 10), (2, 300), (1, 3000), (16, 41)):
        offs = pool.alloc(rung, n)
        assert offs.dtype == np.int64 and offs.size == n and (offs % 512 == 0).all()
        got += [(int(o), int(o) + pool.slot[rung]) for o in offs]
    got.sort()
    assert all(a[1] <= b[0] for a, b in zip(got, got[1:]))
    assert got[-1][1] <= pool.capacity_bytes
    assert pool.bytes_in_use == 91 * 32768 + 90 * 18432 + 10 * 10240 + 300 * 6144 + 3000 * 512


def test_demotion_pattern_returns_bytes_and_slabs():
    pool = make_pool()
    big = pool.alloc(16, 90)                       # two slabs of rung 16
    assert pool.bytes_reserved == 2 * pool.slab_bytes
    small = pool.alloc(4, 90)
    freed_slab = int(big[0]) // pool.slab_bytes
    assert (big[:45] // pool.slab_bytes == freed_slab).all()
    pool.free(16, big[:45])                        # that slab empties and goes back
    assert pool.bytes_reserved == 2 * pool.slab_bytes
    assert pool.bytes_in_use == 45 * 32768 + 90 * 10240
    again = pool.alloc(2, 10)                      # reuses the returned slab for another rung
    assert (again // pool.slab_bytes == freed_slab).all()
    pool.free(16, big[45:])
    pool.free(4, small)
    pool.free(2, again)
    assert pool.bytes_in_use == 0 and pool.bytes_reserved == 0
    assert pool.peak_bytes_in_use == 90 * 32768 + 90 * 10240


def test_exhaustion_and_wrong_rung_are_errors():
    from geodesia_kv_b200.paged import PoolExhausted
    pool = make_pool(mib=3)                        # two slabs
    a = pool.alloc(16, 45)
    pool.alloc(8, 80)
    with pytest.raises(PoolExhausted):
        pool.alloc(4, 1)
    with pytest.raises(ValueError):
        pool.free(8, a[:1])
    pool.free(16, a)
    assert pool.alloc(4, 144).size == 144


class PlainPool:
    """The bookkeeping one slot at a time."""

    def __init__(self, slot, slab_bytes, n_slabs):
        self.slot, self.slab, self.free_slabs = slot, slab_bytes, list(range(n_slabs - 1, -1, -1))
        self.stack, self.rung, self.live = {r: [] for r in slot}, {}, {}

    def alloc(self, rung, n):
        while len(self.stack[rung]) < n:
            s = self.free_slabs.pop()
            self.rung[s], self.live[s] = rung, 0
            self.stack[rung] += [s * self.slab + i * self.slot[rung] for i in reversed(range(self.slab // self.slot[rung]))]
        out = [self.stack[rung].pop() for _ in range(n)]
        for o in out:
            self.live[o // self.slab] += 1
        return out

    def free(self, rung, offs):
        for o in offs:
            self.live[o // self.slab] -= 1
        self.stack[rung] += offs
        for s in sorted({o // self.slab for o in offs if self.live[o // self.slab] == 0}, reverse=True):
            self.stack[rung] = [o for o in self.stack[rung] if o // self.slab != s]
            self.free_slabs.append(s)
            del self.rung[s], self.live[s]


@pytest.mark.parametrize("slabs", [30, 400, 20000])      # below, among and far above the numbers of slots moved
def test_bookkeeping_is_the_plain_one_for_short_and_long_pools(slabs):
    from geodesia_kv_b200.paged import LADDER, PagedPool
    pool = PagedPool(slabs * 1474560, 128, 32, device="meta")
    plain = PlainPool(pool.slot, pool.slab_bytes, slabs)
    rng = np.random.default_rng(slabs)
    held = {r: [] for r in LADDER}
    for _ in range(300):
        rung = int(rng.choice(LADDER))
        n = int(rng.choice([1, 7, 60, 150]))
        if rng.random() < 0.55 and sum(map(len, held.values())) < 800:
            got = pool.alloc(rung, n).tolist()
            assert got == plain.alloc(rung, n)
            held[rung] += got
        elif held[rung]:
            offs = [held[rung].pop(int(rng.integers(len(held[rung])))) for _ in range(min(n, len(held[rung])))]
            pool.free(rung, np.array(offs))
            plain.free(rung, offs)
        assert pool._free_slabs == plain.free_slabs
        assert pool._stack[rung][:pool._top[rung]].tolist() == plain.stack[rung]
        assert pool.slots_in_use(rung) == len(held[rung])
    assert pool.bytes_in_use == sum(len(h) * pool.slot[r] for r, h in held.items())


def test_moving_a_few_slots_does_not_cost_the_length_of_the_pool():
    """Scratch of a few slots' worth, in a pool of 160 GB whose per-slab arrays are 880 KB long."""
    import tracemalloc
    from geodesia_kv_b200.paged import PagedPool
    pool = PagedPool(110_000 * 1474560, 128, 32, device="meta")
    pool.alloc(16, 500)
    tracemalloc.start()
    try:
        for _ in range(3):
            pool.free(16, pool.alloc(16, 16))
            pool.free(16, pool.alloc(16, 100))                  # some slabs empty
        assert tracemalloc.get_traced_memory()[1] < 64 << 10
    finally:
        tracemalloc.stop()


def test_running_out_leaves_the_pool_as_it_was():
    from geodesia_kv_b200.paged import LADDER, PagedLayerCache, PagedPool, PoolExhausted
    pool = PagedPool(4 * 1474560, 128, 32, device="cpu")         # four slabs
    with pytest.raises(PoolExhausted):
        pool.alloc(16, 5 * 45)
    assert pool.bytes_reserved == 0                              # no slab stays behind for the slots refused
    eights = pool.alloc(8, 3 * 80)
    layer = PagedLayerCache(pool, 1, 1)
    layer.offs_h[0, :40], layer.level_h[0, :40], layer.len_h[0] = pool.alloc(16, 40), 16, 40 * 64
    pool.free(8, eights[:10])                                    # ten slots of 8 bits are free, a slab for 4 bits is not
    before, tgt = pool.bytes_in_use, np.zeros((1, 40), dtype=np.int32)
    tgt[0, 10:20], tgt[0, 20:30] = LADDER.index(8), LADDER.index(4)
    with pytest.raises(PoolExhausted):
        layer.apply_demotion(tgt)
    assert pool.bytes_in_use == before and (layer.level_h[0, :40] == 16).all()
    assert pool.alloc(8, 10).size == 10
