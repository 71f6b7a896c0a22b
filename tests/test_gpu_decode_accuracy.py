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


@pytest.mark.parametrize("rep", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("D,group", [(128, 32), (64, 16)])
def test_a_token_that_takes_the_whole_weight_comes_out_as_it_was_stored(ext, rep, D, group):
    """Raw blocks: the largest weight is 1, which its two bf16 halves hold exactly.  The query is 70 to 88 times one
    key of length 1, so the other tokens' weights vanish.  The rounding of an exponent cancels in the division; what is left
    are two truncations, 2^-22.  Weights one rounding of 16 bits off differ by up to 2^-17."""
    from geodesia_kv_b200.pack_layout import pack_cache
    gen = torch.Generator(device="cuda").manual_seed(rep * D)
    T, Hkv = 64 * 12, 2
    k = torch.nn.functional.normalize(torch.randn(1, Hkv, T, D, device="cuda", generator=gen), dim=-1).to(torch.bfloat16)
    v = torch.randn(1, Hkv, T, D, device="cuda", generator=gen).to(torch.bfloat16)
    cache = pack_cache(k, v, torch.full((1, Hkv, T // 64), 16, dtype=torch.int32, device="cuda"), group)
    at = torch.randint(0, T, (Hkv, rep), device="cuda", generator=gen)
    picked = k[0, torch.arange(Hkv, device="cuda")[:, None], at].float()
    q = (picked * torch.linspace(70.0, 88.0, rep, device="cuda")[None, :, None]).reshape(1, Hkv * rep, D).contiguous()
    scores = torch.einsum("hrd,htd->hrt", q.view(Hkv, rep, D).double(), k[0].double())
    rest = torch.softmax(scores, -1).scatter(-1, at[..., None], 0.0).sum(-1).max()
    assert rest < 2.0 ** -24                                   # the case is what it says
    out = ext.mixed_attn_decode(q, *cache.kernel_args()).view(Hkv, rep, D).double()
    want = v[0, torch.arange(Hkv, device="cuda")[:, None], at].double()
    assert ((out - want).norm(dim=-1) / want.norm(dim=-1)).max() < 2.0 ** -21


@pytest.mark.parametrize("T,peak,bound", [(2000, 1.0, 2.0e-7), (16384, 6.0, 3.3e-7)])
@pytest.mark.parametrize("Hq,Hkv", [(16, 2), (4, 4)])
def test_rows_of_centroids_are_as_accurate_as_fp32(ext, T, peak, bound, Hq, Hkv):
    """FP32 arithmetic throughout has 1.2e-7 (one unit of 2^-23) and, with scores six times as large, 2.2e-7; the bounds are one
    and a half times that, over enough rows for the spread to average out."""
    got = []
    for seed in range(12):
        gen, cache = packed(100 + seed, Hkv, T, 128, 32, 1)
        got.append(errors(ext, cache, torch.randn(1, Hq, 128, device="cuda", generator=gen) * (peak * 128 ** -0.5)))
    assert float(torch.stack(got).square().mean().sqrt()) < bound
