"""Edges of the block kernels: tile remainders, alignment, the forms a dispatch sends elsewhere — against the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import oracle_cache, to_torch

pytestmark = pytest.mark.gpu

LADDER = np.array([16, 8, 4, 2, 1], np.int32)


@pytest.mark.parametrize("shift", [0, 2])            # 2: blocks that the wide loads cannot take
@pytest.mark.parametrize("D,group", [(128, 32), (128, 16), (128, 64), (64, 16), (64, 64), (128, 128), (64, 32), (96, 32)])
def test_unpack_every_rung(oracle, D, group, shift):
    from geodesia_kv_b200.pack_layout import PackedCache, unpack_cache
    levels = [16, 4, 2, 1, 8, 2, 4, 16]
    c = oracle_cache(oracle, 70 + D + group, 1, 2, len(levels), D, group, levels=levels)
    c["data"] = np.pad(c["data"], ((0, 0), (0, 0), (shift, 0)))
    c["offs"] = c["offs"] + shift
    t = to_torch(c, "cuda")
    k, v = unpack_cache(PackedCache(t["data"], t["offs"], t["klo"], t["kstep"], t["vlo"], t["vstep"], t["level"], t["valid"], group, D))
    k, v = (x.cpu().numpy().reshape(2, len(levels), 64, D) for x in (k, v))
    for h in range(2):
        for i, lv in enumerate(levels):
            o = int(c["offs"][0, h, i])
            wk, wv = oracle.dequant_block(c["data"][0, h, o:o + oracle.block_bytes(lv, 64, D)], lv, 64, D, group, c["klo"][0, h, i],
                                          c["kstep"][0, h, i], c["vlo"][0, h, i], c["vstep"][0, h, i])
            assert np.array_equal(k[h, i].view(np.uint32), wk.view(np.uint32)), (h, i, lv)
            assert np.array_equal(v[h, i].view(np.uint32), wv.view(np.uint32)), (h, i, lv)


def awkward(seed, shape, kind):
    """kind 0: plain; 1: channels over eight decades; 2: small spreads on large offsets; 3: infinities, NaNs, constant groups."""
    rng = np.random.default_rng(seed)
    nb, P, D = shape
    x = rng.standard_normal(shape).astype(np.float32)
    if kind >= 1:
        x *= np.exp(4 * rng.standard_normal((nb, 1, D))).clip(1e-4, 1e4).astype(np.float32)
    if kind >= 2:
        x = np.where(rng.random(shape) < 0.7, (300 * rng.standard_normal((nb, 1, D)) + 1e-3 * x).astype(np.float32), x)
    if kind >= 3:
        u = rng.random(shape)
        x[u < 0.002] = np.inf
        x[(u > 0.002) & (u < 0.004)] = -np.inf
        x[(u > 0.004) & (u < 0.006)] = np.nan
        x[0] = 3.0
        x[1, :, :16] *= np.float32(1e-7)
    return x


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D,group", [(128, 32), (128, 16), (128, 64), (128, 128), (64, 16), (64, 32), (64, 64)])
def test_pack_awkward_values(oracle, D, group, dtype):
    """Codes near ties, quotients beyond 16 bits, steps that round to zero, values that are not numbers; the last block is short."""
    from geodesia_kv_b200.pack_layout import block_nbytes, pack_cache
    levels = np.array([8, 4, 2, 4, 8, 2, 16, 4], np.int32)
    nb = levels.size
    for kind in range(4):
        T = nb * 64 - (0 if kind == 0 else 40 + kind)
        dense = [torch.from_numpy(awkward(10 * kind + s, (nb, 64, D), kind)).view(nb * 64, D)[:T].to(dtype) for s in (1, 2)]
        cache = pack_cache(*(x.cuda().view(1, 1, T, D) for x in dense), torch.from_numpy(levels).cuda().view(1, 1, nb), group)
        full = [torch.cat([x, x[-1:].expand(nb * 64 - T, D)]).float().numpy().reshape(nb, 64, D) for x in dense]
        want = oracle.pack_row(*full, levels, group)
        assert cache.valid.flatten().tolist() == [64] * (nb - 1) + [64 - (nb * 64 - T)]
        data = cache.data.cpu().numpy()[0, 0]
        assert not data[want["data"].size:].any()
        for i, lv in enumerate(levels):
            if lv == 16 and kind == 3:
                continue                                     # NaN payloads are not defined
            o, n = int(want["offs"][i]), block_nbytes(int(lv), D)
            assert int(cache.offs[0, 0, i]) == o
            assert np.array_equal(data[o:o + n], want["data"][o:o + n]), (kind, i, int(lv))
        for key in ("klo", "kstep", "vlo", "vstep"):
            got, ref = (a.view(np.float16) for a in (getattr(cache, key).cpu().view(torch.int16).numpy().view(np.uint16)[0, 0], want[key]))
            assert np.array_equal(got, ref, equal_nan=True), (kind, key)


@pytest.mark.parametrize("nb", [1, 63, 64, 65, 200])
def test_layout_of_rows(nb):
    from geodesia_kv_b200.pack_layout import layout_offsets, pack_cache
    rng = np.random.default_rng(nb)
    for T in (nb * 64, nb * 64 - 63):
        level = torch.from_numpy(LADDER[rng.integers(0, 5, (2, 2, nb))]).cuda()
        k = torch.randn(2, 2, T, 64, device="cuda", dtype=torch.bfloat16)
        cache = pack_cache(k, k, level, 32)
        offs, row_bytes = layout_offsets(level, 64)
        assert torch.equal(cache.offs, offs) and cache.data.shape[-1] == -(-int(row_bytes.max()) // 256) * 256
        assert cache.valid[..., -1].eq(64 - (nb * 64 - T)).all() and cache.valid[..., :-1].eq(64).all()
        behind = torch.arange(cache.data.shape[-1], device="cuda") >= row_bytes[..., None]
        assert not cache.data[behind].any()


def test_tails_of_unequal_rows():
    """Rows of very different rungs: the tails are zeros, whatever the row count, and cost no more than filling the
    whole buffer a few times over (one CTA per row takes some hundred times as long)."""
    from geodesia_kv_b200.pack_layout import layout_offsets, pack_cache
    for rows, nb in ((1, 3), (2, 2048), (9, 50), (700, 2)):
        level = torch.full((1, rows, nb), 1, dtype=torch.int32, device="cuda")
        level[:, rows // 2] = 16
        level[:, 0, ::2] = 2
        k = torch.randn(1, rows, nb * 64, 128, device="cuda", dtype=torch.bfloat16)
        junk = torch.full((1, rows, nb * 32768), 255, dtype=torch.uint8, device="cuda")
        del junk                                                 # the buffer that follows is likely to hold it
        cache = pack_cache(k, k, level, 32)
        _, row_bytes = layout_offsets(level, 128)
        for r in range(rows if rows < 10 else 20):
            assert not cache.data[0, r, int(row_bytes[0, r]):].any(), (rows, r)
        if nb < 2048:
            continue
        def best(fn):
            times = []
            for _ in range(8):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                fn()
                b.record()
                torch.cuda.synchronize()
                times.append(a.elapsed_time(b))
            return min(times)
        assert best(lambda: pack_cache(k, k, level, 32)) < 10 * best(lambda: cache.data.fill_(0))


@pytest.mark.parametrize("D,group", [(128, 32), (128, 16), (128, 64), (64, 16), (64, 64), (96, 32)])
@pytest.mark.parametrize("value_weight", [0.0, 0.5])
def test_distortion_edges(oracle, D, group, value_weight):
    """The V half enters with weight 0 unless one of its values is too large for that to be 0."""
    from geodesia_kv_b200 import policies
    from geodesia_kv_b200.pack_layout import pack_cache
    nb = 6
    k = torch.from_numpy(awkward(1, (nb, 64, D), 1)).bfloat16()
    v = torch.from_numpy(awkward(2, (nb, 64, D), 1)).bfloat16()
    v[1, 3, 5] = 2.0 ** 41
    v[2, 60, D - 1] = float("inf")
    v[3, 0, 0] = float("nan")
    k[4, 7, 9] = float("inf")
    level = torch.full((1, 1, nb), 16, dtype=torch.int32, device="cuda")
    cache = pack_cache(k.cuda().view(1, 1, -1, D), v.cuda().view(1, 1, -1, D), level, group)
    E = policies.block_distortion(cache, value_weight).cpu().numpy()[0, 0]
    want = oracle.distortion(k.float().numpy(), v.float().numpy(), group, value_weight)
    assert np.array_equal(E, want, equal_nan=True)


@pytest.mark.parametrize("nb", [1, 32, 33, 100, 512, 513])
@pytest.mark.parametrize("whole", [True, False])
def test_allocate_sizes(oracle, nb, whole):
    """A block per thread up to 512, several above; rungs that cost whole bits are added as integers."""
    import ctypes as C
    from geodesia_kv_b200 import _lib
    lib, rows = _lib.load(), 5
    rng = np.random.default_rng(nb)
    E = ((np.abs(rng.standard_normal((rows, nb, 1))) + 0.5) * np.array([0.0, 0.02, 0.3, 1.5, 6.0])).astype(np.float32)
    mass = rng.random((rows, nb), dtype=np.float32)
    idx = np.maximum(rng.integers(-4, 5, (rows, nb)), 0).astype(np.int32)
    hot = (rng.random((rows, nb)) < 0.1).astype(np.uint8)
    bits = np.array([262144, 147456, 81920, 49152, 4096], np.float32) + (0 if whole else 0.25)
    budget = np.array([0.1, 2.5, 4.0, 7.0, 50.0]) * 2 * 64 * 128 * nb
    cu = [torch.from_numpy(a).cuda() for a in (mass, E, idx, hot, budget)]
    ratio, tgt = torch.empty(rows, nb, 4, device="cuda"), torch.empty(rows, nb, dtype=torch.int32, device="cuda")
    rc = lib.gkv_allocate(cu[0].data_ptr(), cu[1].data_ptr(), cu[2].data_ptr(), cu[3].data_ptr(), (C.c_float * 5)(*bits), cu[4].data_ptr(),
                          1.0, ratio.data_ptr(), tgt.data_ptr(), rows, nb, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    for r in range(rows):
        want, ref = oracle.allocate(mass[r], E[r], idx[r], hot[r], bits, budget[r])
        assert np.array_equal(tgt[r].cpu().numpy(), want), (r, nb)
        assert np.array_equal(ratio[r].cpu().numpy(), ref)


@pytest.mark.parametrize("D,group,Hkv,lengths", [(128, 32, 2, [1, 64, 65, 640, 1999]), (64, 32, 1, [33000, 500, 32768]), (64, 16, 2, [32769])])
def test_table_form_plans_as_the_array_form(D, group, Hkv, lengths):
    """The allocator's inputs derived from a ragged block table, against the same inputs spelled out; rows beyond 512 blocks
    keep their ratios in memory."""
    import ctypes as C
    from geodesia_kv_b200 import _lib, policies
    from geodesia_kv_b200.paged import PagedLayerCache, PagedPool
    lib, B = _lib.load(), len(lengths)
    layer = PagedLayerCache(PagedPool(64 << 20, D, group), B, Hkv)
    k = torch.randn(B, Hkv, max(lengths), D, device="cuda", dtype=torch.bfloat16)
    layer.prefill(k, k, lengths)
    mass = torch.rand(layer.rows, layer.nb + 3, device="cuda")                # wider than the table is used
    stream = torch.cuda.current_stream().cuda_stream
    for step in range(2):                                                     # the second time some blocks have moved
        nb, rows = layer.nb, layer.rows
        got = layer.plan_demotion(4.0, mass=mass)
        level = layer.level[:, :nb].contiguous()
        idx = ((level <= 8).int() + (level <= 4).int() + (level <= 2).int() + (level <= 1).int()).contiguous()
        E = torch.empty(rows, nb, 5, device="cuda")
        offs, m, hot = layer.offs[:, :nb].contiguous(), mass[:, :nb].contiguous(), layer.hot_blocks(nb)
        assert lib.gkv_block_distortion(layer.pool.data.data_ptr(), offs.data_ptr(), level.data_ptr(), E.data_ptr(),
                                        rows, nb, D, 64, group, 0.0, 0, rows, stream) == 0
        nb_of = ((layer.lens + 63) // 64).int().contiguous()
        target = nb_of.double() * (4.0 * 2.0 * 64 * D)
        ratio, want = torch.empty(rows, nb, 4, device="cuda"), torch.empty(rows, nb, dtype=torch.int32, device="cuda")
        bits = (C.c_float * 5)(*policies.ladder_bits(64, D, group))
        assert lib.gkv_allocate_ragged(m.data_ptr(), E.data_ptr(), idx.data_ptr(), hot.data_ptr(), bits,
                                       target.data_ptr(), 1.0, ratio.data_ptr(), want.data_ptr(), nb_of.data_ptr(), rows, nb, stream) == 0
        assert torch.equal(got, want), step
        assert step or layer.apply_demotion(got.cpu().numpy()) > 0


@pytest.mark.parametrize("B,Hkv", [(3, 2), (1, 1)])
def test_plan_takes_mass_in_every_shape(B, Hkv):
    """What the decode calls return, flat values, wider rows, other types and strides: the plan of the plain (rows, nb)."""
    from geodesia_kv_b200.paged import PagedLayerCache, PagedPool
    nb, rows = 20, B * Hkv
    layer = PagedLayerCache(PagedPool(64 << 20, 64, 32), B, Hkv)
    k = torch.randn(B, Hkv, nb * 64, 64, device="cuda", dtype=torch.bfloat16)
    layer.prefill(k, k)
    m = torch.rand(rows, nb, device="cuda")
    want = layer.plan_demotion(4.0, mass=m)
    assert (want > 0).any()
    wide, spread = torch.rand(rows, nb + 9, device="cuda"), torch.zeros(rows, nb, 3, device="cuda")
    wide[:, :nb], spread[..., 1] = m, m
    for form in (m.view(B, Hkv, nb), m.view(-1), m.view(B, Hkv * nb), wide, wide[:, :nb], m.double(), wide.double(), m.t().contiguous().t(), spread[..., 1]):
        assert torch.equal(layer.plan_demotion(4.0, mass=form), want), (tuple(form.shape), form.stride())
    assert torch.equal(layer.plan_demotion(4.0, mass=m[:1]), layer.plan_demotion(4.0, mass=m[0]))
    with pytest.raises(RuntimeError):
        layer.plan_demotion(4.0, mass=m[:, :-1])


@pytest.mark.parametrize("B,Hq,Hkv", [(1, 7, 1), (200, 8, 8), (120, 8, 2), (64, 64, 8), (3, 12, 4), (40, 16, 2),
                                      (296, 1, 1), (297, 1, 1), (740, 1, 1), (741, 1, 1), (1628, 1, 1), (1629, 1, 1)])
def test_merge_widths_and_mass(oracle, B, Hq, Hkv):
    """From 7 to 4096 output rows the merge runs with 8, 4, 2 and 1 warps per row, on 148 SMs up to 296, 740 and 1628 rows and
    beyond; the mass takes 1 to 8 heads per cache row.

    Both are sums of fp32 products whose operands carry 22 bits: 5e-5 absolute is what the kernel states for outputs of
    order one, masses are sums of weights that add up to one."""
    from geodesia_kv_b200.cuda_ext import get_ext
    from geodesia_kv_b200.pack_layout import pack_cache
    nb, D, group = 9, 64, 32
    gen = torch.Generator(device="cuda").manual_seed(B + Hq)
    k, v = (torch.randn(B, Hkv, nb * 64 - 5, D, device="cuda", generator=gen) for _ in range(2))
    level = torch.from_numpy(LADDER).cuda()[torch.randint(0, 5, (B, Hkv, nb), device="cuda", generator=gen)]
    cache = pack_cache(k, v, level, group)
    q = torch.randn(B, Hq, D, device="cuda", generator=gen) * D ** -0.5
    ext = get_ext()
    out, mass = ext.mixed_attn_decode_with_mass(q, *cache.kernel_args())
    plain = ext.mixed_attn_decode(q, *cache.kernel_args())
    ext.set_decode_kernel("generic")
    try:
        want = ext.mixed_attn_decode(q, *cache.kernel_args())
    finally:
        ext.set_decode_kernel("auto")
    assert (out - want).abs().max() < 5e-5 and (plain - want).abs().max() < 5e-5
    assert (mass.sum(-1) - 1).abs().max() < 1e-5
    one = [t[:1].contiguous().cpu() for t in (q, cache.data, cache.offs, cache.klo, cache.kstep, cache.vlo, cache.vstep, cache.level, cache.valid)]
    arrays = [t.view(torch.int16).numpy().view(np.uint16) if t.dtype == torch.float16 else t.numpy() for t in one]
    assert np.abs(mass[:1].cpu().numpy() - oracle.block_mass(*arrays, 64, group)).max() < 1e-5


def _pool_blocks(rng, D, group, levels, slot):
    """Packed blocks with values and scales of every size, `slot` bytes apart; the bytes behind a block stay as they are."""
    n, G, gv = levels.size, 64 // min(group, 64), D // min(group, D)
    pool = rng.integers(0, 256, (n, slot), dtype=np.uint8)
    for i, lv in enumerate(levels):
        nbytes = 4 * 64 * D if lv == 16 else 64 * D * int(lv) // 4
        if lv == 16:
            x = torch.from_numpy(rng.standard_normal(2 * 64 * D).astype(np.float32)).bfloat16()
            pool[i, :nbytes] = x.view(torch.int16).numpy().view(np.uint8)
        else:
            scales = (rng.random(2 * (G * D + 64 * gv)).astype(np.float16) + np.float16(0.01)).view(np.uint8)
            pool[i, nbytes:nbytes + scales.size] = scales
    return pool


@pytest.mark.parametrize("D,group", [(128, 32), (64, 16)])
def test_stages_shared_by_packed_and_exact_blocks(D, group):
    """A stage of the ring holds blocks of every source rung in turn, copied in or brought in by hand (the pool that
    starts 8 bytes off), and a packed block's partial ranges in between: the same bytes as when no stage is used twice."""
    from geodesia_kv_b200 import _lib
    lib, slot, n = _lib.load(), 512 * D, 4000                   # a CTA has four blocks or more, two per stage
    rng = np.random.default_rng(D)
    old = np.array([8, 16, 4, 16, 8, 16, 16], np.int32)[np.arange(n) % 7]
    new = np.array([4, 4, 2, 1, 2, 8, 2], np.int32)[np.arange(n) % 7]
    pool = torch.from_numpy(_pool_blocks(rng, D, group, old, slot)).cuda()
    off = torch.arange(n, device="cuda") * slot
    lo, ln = torch.from_numpy(old).cuda(), torch.from_numpy(new).cuda()
    stream = torch.cuda.current_stream().cuda_stream

    def demote(shift, per_launch):
        src = torch.zeros(n * slot + 16, dtype=torch.uint8, device="cuda")
        src[shift:shift + n * slot] = pool.view(-1)
        dst, ek, ev = torch.zeros(n * slot, dtype=torch.uint8, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
        for i in range(0, n, per_launch):
            m = min(per_launch, n - i)
            assert lib.gkv_paged_demote_blocks(src.data_ptr() + shift, off[i:].data_ptr(), lo[i:].data_ptr(), dst.data_ptr(), off[i:].data_ptr(),
                                               ln[i:].data_ptr(), ek[i:].data_ptr(), ev[i:].data_ptr(), m, D, 64, group, stream) == 0
        return dst, ek, ev

    want = demote(0, 64)                                         # every CTA has one block
    for shift in (0, 8):
        for got, ref in zip(demote(shift, n), want):
            assert torch.equal(got, ref), shift


def test_stages_shared_by_rows_copied_and_rows_brought_by_hand():
    """Every second block's rows start at an address that a copy cannot take."""
    from geodesia_kv_b200 import _lib
    lib, D, group, n = _lib.load(), 128, 32, 4000
    k, v = (torch.randn(n * 64 * D + 8, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    src = torch.arange(n, device="cuda") * (64 * D) + (torch.arange(n, device="cuda") % 2) * 3
    level = torch.tensor([8, 4, 2, 1, 16], dtype=torch.int32, device="cuda")[torch.arange(n, device="cuda") % 5].contiguous()
    slots = torch.arange(n, device="cuda") * (256 * D)
    stream = torch.cuda.current_stream().cuda_stream

    def pack(per_launch):
        pool = torch.zeros(n * 256 * D, dtype=torch.uint8, device="cuda")
        for i in range(0, n, per_launch):
            m = min(per_launch, n - i)
            assert lib.gkv_paged_pack_blocks(k.data_ptr(), v.data_ptr(), 1, src[i:].data_ptr(), D, None, pool.data_ptr(), slots[i:].data_ptr(),
                                             level[i:].data_ptr(), None, None, m, D, 64, group, stream) == 0
        return pool

    assert torch.equal(pack(n), pack(64))


@pytest.mark.parametrize("D,group,Hq", [(128, 32, 8), (64, 16, 2)])
def test_decode_ring_of_short_and_hand_copied_blocks(oracle, D, group, Hq):
    """Every region of the byte rings holds copied blocks, blocks at odd addresses brought in by hand, scale planes, and
    short blocks whose tails are cleared in place, one after the other.

    5e-5: the kernel's stated error for outputs of order one (operands carry 22 bits)."""
    from geodesia_kv_b200.cuda_ext import get_ext
    from helpers import kernel_args, oracle_args
    Hkv, nb = 2, 700
    c = oracle_cache(oracle, 900 + D, 1, Hkv, nb, D, group, probs=(0.2, 0.25, 0.25, 0.2, 0.1))
    rng = np.random.default_rng(D)
    c["valid"][:] = np.where(rng.random(c["valid"].shape) < 0.5, rng.integers(1, 65, c["valid"].shape), 64)
    sizes = np.array([[oracle.block_bytes(int(lv), 64, D) for lv in c["level"][0, h]] for h in range(Hkv)])
    moved = np.where(np.arange(nb) % 3 == 0, 4, 0)[None] + 16 * np.arange(nb)[None] + c["offs"][0]      # every third at an odd address
    data = np.zeros((1, Hkv, int((moved + sizes).max()) + 64), np.uint8)
    for h in range(Hkv):
        for i in range(nb):
            o, m, n = int(c["offs"][0, h, i]), int(moved[h, i]), int(sizes[h, i])
            data[0, h, m:m + n] = c["data"][0, h, o:o + n]
    c["data"], c["offs"] = data[..., :data.shape[-1] // 16 * 16].copy(), moved[None].astype(np.int64)
    t = to_torch(c, "cuda")
    q = rng.standard_normal((1, Hq, D), dtype=np.float32) * np.float32(D ** -0.5)
    got = get_ext().mixed_attn_decode(torch.from_numpy(q).cuda(), *kernel_args(t, c)).cpu().numpy()
    assert np.abs(got - oracle.mixed_attn_decode(q, *oracle_args(c))).max() < 5e-5
    assert get_ext().decode_status() == 0


@pytest.mark.parametrize("D,group,Hq", [(128, 32, 14), (64, 16, 6), (128, 64, 2)])
def test_queries_at_any_address(oracle, D, group, Hq):
    """Queries that start 4, 8 or 12 bytes off a 16-byte boundary are read element by element: the same numbers.

    5e-5: the kernel's stated error for outputs of order one."""
    from geodesia_kv_b200.cuda_ext import get_ext
    from helpers import kernel_args, oracle_args
    c = oracle_cache(oracle, 77 + D, 3, 2, 13, D, group, last_valid=21)
    t = to_torch(c, "cuda")
    q = np.random.default_rng(D).standard_normal((3, Hq, D), dtype=np.float32) * np.float32(D ** -0.5)
    want = oracle.mixed_attn_decode(q, *oracle_args(c))
    for shift in (1, 2, 3):
        buf = torch.full((q.size + 8,), float("nan"), device="cuda")
        buf[shift:shift + q.size] = torch.from_numpy(q).cuda().view(-1)
        view = buf[shift:shift + q.size].view(3, Hq, D)
        assert view.data_ptr() % 16 == 4 * shift
        out, mass = get_ext().mixed_attn_decode_with_mass(view, *kernel_args(t, c))
        for got in (out, get_ext().mixed_attn_decode(view, *kernel_args(t, c))):
            assert np.abs(got.cpu().numpy() - want).max() < 5e-5, shift
        assert (mass.sum(-1) - 1).abs().max() < 1e-5


def test_decode_from_two_streams():
    """Block lists made on one stream and used on another before they are finished; eager work before, between and
    after calls whose launches overlap."""
    from geodesia_kv_b200.cuda_ext import get_ext
    from geodesia_kv_b200.pack_layout import pack_cache
    ext, D, group, Hkv, nb = get_ext(), 128, 32, 2, 70
    gen = torch.Generator(device="cuda").manual_seed(8)
    k = torch.randn(2, Hkv, nb * 64 - 9, D, device="cuda", generator=gen)
    level = torch.from_numpy(LADDER).cuda()[torch.randint(0, 5, (2, Hkv, nb), device="cuda", generator=gen)]
    q = torch.randn(2, 8, D, device="cuda", generator=gen) * D ** -0.5
    cache = pack_cache(k, k, level, group)
    scales = [0.25 * (i + 1) for i in range(12)]
    want = [ext.mixed_attn_decode(q * x, *cache.kernel_args()) + x for x in scales]
    fresh = pack_cache(k, k, level, group)                       # the same metadata at new addresses: no lists yet
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    got = [[], []]
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(100_000_000)                           # the lists wait behind some 50 ms of other work
    for x in scales:
        for s, outs in zip(streams, got):
            with torch.cuda.stream(s):
                scaled = q * x
                out = ext.mixed_attn_decode(scaled, *fresh.kernel_args())
                scaled.fill_(float("nan"))                       # queued behind the call that reads it
                outs.append(out.add_(x))
    torch.cuda.synchronize()
    for outs in got:
        for a, b in zip(outs, want):
            assert (a - b).abs().max() < 5e-5                    # the kernel's stated error; the order of records varies


@pytest.mark.parametrize("same_stream", [True, False])
def test_a_graph_keeps_the_block_lists_it_was_captured_with(monkeypatch, same_stream):
    """Lists that leave the cache of recent metadata stay for a graph that reads them, until its metadata goes."""
    import gc
    from geodesia_kv_b200.cuda_ext import get_ext
    from geodesia_kv_b200.pack_layout import pack_cache
    ext, nb, D = get_ext(), 40, 64
    monkeypatch.setattr(ext, "PLAN_CACHE_ENTRIES", 2)
    gc.collect()
    before = len(ext._captured)
    level = torch.from_numpy(LADDER).cuda()[torch.randint(0, 5, (1, 2, nb), device="cuda")]
    k, q = torch.randn(1, 2, nb * 64, D, device="cuda"), torch.randn(1, 4, D, device="cuda") * D ** -0.5
    caches = [pack_cache(k, k, level, 32) for _ in range(4)]
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = ext.mixed_attn_decode(q, *caches[0].kernel_args())
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side if same_stream else torch.cuda.Stream()):
        out = ext.mixed_attn_decode(q, *caches[0].kernel_args())
    assert len(ext._captured) == before + 1
    kept = list(ext._captured.values())[-1]
    lists = kept.clone()
    for c in caches[1:]:
        ext.mixed_attn_decode(q, *c.kernel_args())               # the cache of lists holds two entries
    assert not any(kept is plan for entry in ext._plans.values() for plan in entry[0].values())
    torch.cuda.synchronize()
    assert torch.equal(kept, lists)
    graph.replay()
    torch.cuda.synchronize()
    assert (out - want).abs().max() < 5e-5
    del graph, caches, c, out
    ext.invalidate_plans()
    gc.collect()
    assert len(ext._captured) == before
