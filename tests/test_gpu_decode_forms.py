"""Forms of a decode call that share the split kernel's records and plane copies: the exchange merge, and the mass by-product with
one metadata vector for all rows."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    from geodesia_kv_b200.cuda_ext import get_ext
    e = get_ext()
    assert e is not None, "CUDA extension must load on a GPU box"
    e.set_decode_item_blocks(0)
    return e


def packed(seed, B, Hkv, nb, D, group, shared=False):
    from geodesia_kv_b200.pack_layout import pack_cache
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, v = (torch.randn(B, Hkv, 64 * nb - 9, D, device="cuda", generator=gen) for _ in range(2))
    pick = torch.randint(0, 5, (nb,) if shared else (B, Hkv, nb), device="cuda", generator=gen)
    return gen, pack_cache(k, v, torch.tensor([16, 8, 4, 2, 1], dtype=torch.int32, device="cuda")[pick], group)


@pytest.mark.parametrize("D,group", [(128, 32), (64, 16), (96, 32)])       # 96: the CUDA-core kernel
@pytest.mark.parametrize("B,Hkv,rep,nb", [(1, 2, 8, 3), (3, 2, 1, 70), (1, 2, 7, 700)])    # one merge level, and two
def test_the_exchange_merge_of_a_single_rank_is_the_ordinary_merge(ext, D, group, B, Hkv, rep, nb):
    """A world of one: the kernel stores its record into its own inbox and reads it back, nothing else is waited for.  Both merges
    add the same records in FP32; a term passes at most 32 roundings of 2^-24."""
    from geodesia_kv_b200.distributed import SequenceSplitDecoder
    gen, c = packed(nb + D, B, Hkv, nb, D, group)
    dec = SequenceSplitDecoder(B, Hkv * rep, D, "cuda")
    assert dec.available and dec.world == 1
    for ws in ext._workspaces.values():
        ws.fill_(0xff)                                                     # records that nothing writes hold anything
    for _ in range(3):                                                     # two inbox buffers take turns
        q = torch.randn(B, Hkv * rep, D, device="cuda", generator=gen) * D ** -0.5
        want = ext.mixed_attn_decode(q, *c.kernel_args())
        out = dec(q, c)
        assert torch.isfinite(out).all()
        assert (out - want).abs().max() <= 32 * 2.0 ** -24 * largest(want)
    assert dec.status() == 0 and dec.seq.tolist() == [3] * (B * Hkv * rep)


def largest(t):
    return float(t.abs().max())


@pytest.mark.parametrize("D,group", [(128, 16), (128, 32), (128, 64), (64, 16), (64, 32), (64, 64)])
@pytest.mark.parametrize("rep", [1, 7])
@pytest.mark.parametrize("shared", [False, True])
def test_mass_is_the_same_whichever_way_the_planes_arrive(ext, D, group, rep, shared):
    gen, c = packed(D + group, 3, 2, 61, D, group, shared)
    offs, level, valid = ((t[0, 0].contiguous() if shared else t) for t in (c.offs, c.level, c.valid))
    at = [p.data_ptr() for p in (c.klo, c.kstep, c.vlo, c.vstep)]
    assert at[1] - at[0] == at[2] - at[1] == at[3] - at[2] > 0             # one tiled copy per block
    room = torch.empty(2 * c.klo.numel() + 1024, dtype=torch.float16, device="cuda")
    apart = [t.clone() for t in (c.klo, c.kstep, c.vlo)] + [room[8 * 53:8 * 53 + c.vstep.numel()].view(c.vstep.shape).copy_(c.vstep)]
    q = torch.randn(3, 2 * rep, D, device="cuda", generator=gen) * D ** -0.5
    one, mass_one = ext.mixed_attn_decode_with_mass(q, c.data, offs, c.klo, c.kstep, c.vlo, c.vstep, level, valid, 64, group)
    two, mass_two = ext.mixed_attn_decode_with_mass(q, c.data, offs, *apart, level, valid, 64, group)
    plain = ext.mixed_attn_decode(q, c.data, offs, c.klo, c.kstep, c.vlo, c.vstep, level, valid, 64, group)
    assert torch.equal(one, two) and torch.equal(mass_one, mass_two)
    # the variant with the mass is another instantiation of the same arithmetic
    assert (one - plain).abs().max() <= 32 * 2.0 ** -24 * largest(plain)
    assert (mass_one.view(6, -1).sum(1) - 1).abs().max() < 1e-4 and (mass_one >= 0).all()
