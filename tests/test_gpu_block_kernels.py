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
