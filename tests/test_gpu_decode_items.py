"""The tensor-core kernel's work split: items on both sides of the lengths at which blocks and centroid tiles change hands."""
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
