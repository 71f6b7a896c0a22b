"""Attention outputs against 64 bits, relative to the result: means over long sequences are small against their terms, which
a bound on the absolute error does not see."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    from geodesia_kv_b200.cuda_ext import get_ext
    e = get_ext()
    assert e is not None, "CUDA extension must load on a GPU box"
    return e


def packed(seed, Hkv, T, D, group, rung, outliers=4):
    from geodesia_kv_b200.pack_layout import pack_cache
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, v = (torch.randn(1, Hkv, T, D, device="cuda", generator=gen, dtype=torch.bfloat16) for _ in range(2))
    k[..., :outliers] *= 8.0
    return gen, pack_cache(k, v, torch.full((1, Hkv, (T + 63) // 64), rung, dtype=torch.int32, device="cuda"), group)


def errors(ext, cache, q):
    """(B, Hq): distance from attention in 64 bits over the dequantised cache, relative to its norm."""
    from geodesia_kv_b200.pack_layout import unpack_cache
    k, v = unpack_cache(cache)
    B, Hkv, T, _ = k.shape
    rep = q.shape[1] // Hkv
    at = torch.arange(T, device="cuda")
    out = ext.mixed_attn_decode(q, *cache.kernel_args()).double()
    err = torch.empty(q.shape[:2], dtype=torch.float64)
    for b in range(B):
        for h in range(Hkv):
            dead = at % 64 >= cache.valid.view(B, Hkv, -1)[b, h][at // 64]
            mine = slice(h * rep, (h + 1) * rep)
            s = (q[b, mine].double() @ k[b, h].double().T).masked_fill(dead, -torch.inf)
            want = torch.softmax(s, -1) @ v[b, h].double()
            err[b, mine] = ((out[b, mine] - want).norm(dim=-1) / want.norm(dim=-1)).cpu()
    return err


def test_a_long_8_bit_row_is_as_accurate_for_eight_heads_as_for_four(ext):
    """Both add the same products, two roundings of an output to two of its bias for eight heads, one to one for four.  Their
    errors are drifts of the same size; 1.6 leaves room for the spread between rows."""
    eight, four = [], []
    for seed in range(3):
        gen, cache = packed(seed, 1, 1 << 20, 128, 32, 8)
        q = torch.randn(1, 8, 128, device="cuda", generator=gen) * 128 ** -0.5
        eight.append(errors(ext, cache, q))
        four.append(torch.cat([errors(ext, cache, q[:, h:h + 4].contiguous()) for h in (0, 4)], 1))
        del cache
    rms = lambda e: float(torch.stack(e).square().mean().sqrt())
    assert rms(eight) < 1.6 * rms(four)
