"""The tensor-core kernel's work split: items on both sides of the lengths at which blocks and centroid tiles change hands, and
both ways in which the scale planes arrive."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import kernel_args, oracle_args, oracle_cache, to_torch

pytestmark = pytest.mark.gpu
TOL = 5e-5          # fp32 sums over exactly dequantised values, small operands in two 16-bit halves


@pytest.fixture(scope="module")
def ext():
    from geodesia_kv_b200.cuda_ext import get_ext
    e = get_ext()
    assert e is not None, "CUDA extension must load on a GPU box"
    yield e
    e.set_decode_item_blocks(0)


def attend(ext, oracle, c, Hq, seed=3):
    q = np.random.default_rng(seed).standard_normal((c["B"], Hq, c["D"]), dtype=np.float32) * np.float32(c["D"] ** -0.5)
    t = to_torch(c, "cuda")
    out, mass = ext.mixed_attn_decode_with_mass(torch.from_numpy(q).cuda(), *kernel_args(t, c))
    plain = ext.mixed_attn_decode(torch.from_numpy(q).cuda(), *kernel_args(t, c))
    want = oracle.mixed_attn_decode(q, *oracle_args(c))
    assert np.abs(plain.cpu().numpy() - want).max() < TOL and np.abs(out.cpu().numpy() - want).max() < TOL
    rows = c["B"] * c["Hkv"]
    assert np.abs(mass.view(rows, -1).sum(1).cpu().numpy() - 1).max() < 1e-4


@pytest.mark.parametrize("rep", [1, 4, 5, 8])
@pytest.mark.parametrize("blocks,nb", [(23, 23), (24, 24), (25, 51), (128, 130)])
@pytest.mark.parametrize("D,group", [(128, 32), (128, 16), (64, 64)])
def test_items_around_the_length_from_which_a_warp_takes_whole_blocks(ext, oracle, rep, blocks, nb, D, group):
    ext.set_decode_item_blocks(blocks)
    for rung in (8, 4, 2):
        attend(ext, oracle, oracle_cache(oracle, nb + rung, 1, 2, nb, D, group, last_valid=37, levels=[rung] * nb), 2 * rep)


@pytest.mark.parametrize("rep", [1, 8])
@pytest.mark.parametrize("nb", [1, 15, 16, 17, 129, 300])
@pytest.mark.parametrize("D,group", [(128, 32), (64, 16)])
def test_centroid_items_around_a_tile(ext, oracle, rep, nb, D, group):
    ext.set_decode_item_blocks(0)
    attend(ext, oracle, oracle_cache(oracle, nb, 1, 2, nb, D, group, last_valid=5, levels=[1] * nb), 2 * rep)


@pytest.mark.parametrize("D,group", [(128, 16), (128, 32), (128, 64), (64, 16), (64, 32), (64, 64)])
@pytest.mark.parametrize("rep", [2, 7])
def test_planes_at_equal_distances_and_apart_give_the_same_bits(ext, rep, D, group):
    from geodesia_kv_b200.pack_layout import pack_cache
    ext.set_decode_item_blocks(0)
    g = torch.Generator(device="cuda").manual_seed(D + group)
    k, v = (torch.randn(2, 2, 64 * 60 - 9, D, device="cuda", generator=g) for _ in range(2))
    level = torch.tensor([16, 8, 4, 2, 1], dtype=torch.int32, device="cuda")[torch.randint(0, 5, (2, 2, 60), device="cuda", generator=g)]
    c = pack_cache(k, v, level, group)
    at = [p.data_ptr() for p in (c.klo, c.kstep, c.vlo, c.vstep)]
    assert at[1] - at[0] == at[2] - at[1] == at[3] - at[2] > 0
    q = torch.randn(2, 2 * rep, D, device="cuda", generator=g) * D ** -0.5
    one = ext.mixed_attn_decode(q, *c.kernel_args())
    pool = torch.empty(5 * c.klo.numel() + 1024, dtype=torch.float16, device="cuda")
    n, apart = c.klo.numel(), []
    for i, p in zip((3, 0, 2, 1), (c.klo, c.kstep, c.vlo, c.vstep)):        # the same planes in another order
        apart.append(pool[i * n:(i + 1) * n].view(p.shape).copy_(p))
    two = ext.mixed_attn_decode(q, c.data, c.offs, *apart, c.level, c.valid, 64, group)
    odd = pool[4 * n:5 * n + 8]                                             # one plane at an address of its own
    three = ext.mixed_attn_decode(q, c.data, c.offs, c.klo, c.kstep, c.vlo, odd[8:].view(c.vstep.shape).copy_(c.vstep), c.level, c.valid, 64, group)
    assert torch.equal(one, two) and torch.equal(one, three)


@pytest.mark.parametrize("nb", [419, 420, 421, 427])       # two rows: 148 item slots up to 420 blocks, 150 and 152 beyond
def test_calls_around_one_item_slot_per_cta_start_from_any_scratch(ext, oracle, nb):
    ext.set_decode_item_blocks(6)
    c = oracle_cache(oracle, nb, 1, 2, nb, 128, 32, last_valid=11)
    attend(ext, oracle, c, 8)
    for ws in ext._workspaces.values():
        ws.fill_(0xff)                                       # counter and status word hold anything before a call
    attend(ext, oracle, c, 8)
    assert ext.decode_status() == 0
