"""Caches with more tile rows than a 32-bit coordinate counts."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,group,gib", [(64, 32, 66), (64, 16, 66), (128, 32, 130)])
def test_blocks_beyond_the_last_row_that_a_coordinate_reaches(D, group, gib):
    """4-bit blocks are fetched as rows of 32 bytes at D = 64 (2^31 of them end at 64 GiB) and of 64 bytes at D = 128 (at
    128 GiB).  The same blocks at the start and at the end of a pool give the same bits."""
    from geodesia_kv_b200.paged import LADDER, PagedLayerCache, PagedPool
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < (gib + 6) << 30:
        pytest.skip("not enough free device memory")
    pool = PagedPool(64 << 20, D, group)
    layer = PagedLayerCache(pool, 2, 2)
    gen = torch.Generator(device="cuda").manual_seed(D)
    k, v = (torch.randn(2, 2, 64 * 30, D, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2))
    layer.prefill(k, v, [64 * 30, 64 * 11 + 5])
    layer.apply_demotion(np.random.default_rng(D).integers(0, 5, (4, layer.nb)))
    assert set(layer.level_h[layer.level_h > 0]) == set(LADDER)
    q = torch.randn(2, 8, D, device="cuda", generator=gen) * D ** -0.5
    want = layer.attend(q)
    small = pool.data
    pool.data = torch.empty(gib << 30, dtype=torch.uint8, device="cuda")
    shift = (pool.data.numel() - small.numel()) // 256 * 256
    pool.data[shift:shift + small.numel()] = small
    layer.offs = torch.where(layer.offs >= 0, layer.offs + shift, layer.offs)
    out = layer.attend(q)
    torch.cuda.synchronize()
    del pool.data
    torch.cuda.empty_cache()
    assert torch.isfinite(want).all() and torch.equal(out, want)
