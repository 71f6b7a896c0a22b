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
