"""Host bookkeeping of the block table (native) against the same steps in numpy, one array operation at a time."""
import numpy as np
import pytest

from geodesia_kv_b200.paged import LADDER, PagedLayerCache, PagedPool, PoolExhausted, _addr

P = 64


def enter(c, first, count, T, tokens):
    n = int(np.sum(count)) * c.Hkv
    out = [np.full(n, -7, t) for t in (np.int64,) * 3 + (np.int32,) * 3]
    first, count = np.array(first, dtype=np.int64), np.array(count, dtype=np.int64)
    tokens = None if tokens is None else np.array(tokens, dtype=np.int64)
    rc = c.lib.gkv_table_enter(c.pool.handle, _addr(c.offs_h), _addr(c.level_h), c.B, c.Hkv, c.cap, T, c.D, _addr(first), _addr(count),
                               None if tokens is None else _addr(tokens), *map(_addr, out))
    c.pool._check(rc, "test")
    return out


@pytest.mark.parametrize("B,Hkv", [(1, 1), (3, 2), (5, 4)])
@pytest.mark.parametrize("reserved", [False, True])
def test_entering_demoting_and_releasing_follow_numpy(B, Hkv, reserved):
    rng = np.random.default_rng(B * 10 + Hkv)
    pool, other = (PagedPool(20 * 1474560, 128, 32, device="cpu") for _ in range(2))
    c = PagedLayerCache(pool, B, Hkv, cap_blocks=12)
    offs, level = c.offs_h.copy(), c.level_h.copy()
    if reserved:                                            # some entries hold a slot before a token reaches them
        c.offs_h[:, 1], c.level_h[:, 1] = pool.alloc(16, c.rows), 16
        offs[:, 1], level[:, 1] = other.alloc(16, c.rows), 16
    tokens = rng.integers(1, 9 * P, B)
    count, T = (tokens + P - 1) // P, int(tokens.max())
    so, sl, at, nv, lv, rl = enter(c, np.zeros(B), count, T, tokens)
    row = np.repeat(np.arange(c.rows), np.repeat(count, Hkv))
    blk = np.concatenate([np.arange(n) for n in np.repeat(count, Hkv)])
    want = offs[row, blk]
    want[want < 0] = other.alloc(16, int((want < 0).sum()))
    offs[row, blk], level[row, blk] = want, 16
    assert (sl == want).all() and (at == row * c.cap + blk).all() and (so == (row * T + blk * P) * c.D).all()
    assert (nv == np.minimum(P, tokens[row // Hkv] - blk * P)).all() and (lv == 16).all() and (rl == tokens[row // Hkv]).all()
    assert (c.offs_h == offs).all() and (c.level_h == level).all()
    # demotion of a random half, targets out of range included; entries beyond a row's blocks never move
    nb = int(count.max())
    tgt = rng.integers(-1, 7, (c.rows, nb)).astype(np.int32)
    count64 = count.astype(np.int64)
    table = (_addr(c.offs_h), _addr(c.level_h), B, Hkv, c.cap, _addr(count64), _addr(tgt), nb)
    new = np.array(LADDER)[np.clip(tgt, 0, 4)]
    r, b = np.nonzero((new < level[:, :nb]) & (np.arange(nb)[None] < np.repeat(count, Hkv)[:, None]) & (offs[:, :nb] >= 0))
    n = c.lib.gkv_table_demotions(*table)
    assert n == r.size
    old, got, flat, lo, ln = (np.empty(n, t) for t in (np.int64, np.int64, np.int64, np.int32, np.int32))
    c.pool._check(c.lib.gkv_table_plan_demotion(pool.handle, *table, n, *map(_addr, (old, got, flat, lo, ln))), "test")
    want = np.empty(n, np.int64)
    for rung in LADDER[1:]:
        sel = np.nonzero(new[r, b] == rung)[0]
        want[sel] = other.alloc(rung, sel.size)
    assert (old == offs[r, b]).all() and (got == want).all() and (flat == r * c.cap + b).all()
    assert (lo == level[r, b]).all() and (ln == new[r, b]).all() and (c.offs_h == offs).all()
    c.pool._check(c.lib.gkv_table_apply_demotion(pool.handle, *table[:2], n, *map(_addr, (old, got, flat, lo, ln))), "test")
    other.free(16, old)
    offs[r, b], level[r, b] = want, new[r, b]
    assert (c.offs_h == offs).all() and (c.level_h == level).all()
    for rung in LADDER:
        assert pool._stack[rung].tolist() == other._stack[rung].tolist()
    assert pool._free_slabs == other._free_slabs and pool.bytes_in_use == other.bytes_in_use
    assert c.lib.gkv_table_release(pool.handle, _addr(c.offs_h), _addr(c.level_h), c.offs_h.size) == 0
    assert pool.bytes_in_use == 0 and (c.offs_h == -1).all() and (c.level_h == 0).all() and len(pool._free_slabs) == pool.n_slabs


def test_a_table_that_does_not_fit_is_refused_whole():
    pool = PagedPool(1474560, 128, 32, device="cpu")        # one slab: 45 exact slots
    c = PagedLayerCache(pool, 1, 1, cap_blocks=60)
    with pytest.raises(PoolExhausted):
        enter(c, [0], [46], 46 * P, [46 * P])
    assert pool.bytes_reserved == 0 and (c.offs_h == -1).all()
    enter(c, [0], [45], 45 * P, [45 * P])
    with pytest.raises(ValueError):
        enter(c, [45], [16], 16 * P, None)                  # beyond the table
    with pytest.raises(ValueError):
        pool.free(16, np.array([1474560]))                  # beyond the pool
