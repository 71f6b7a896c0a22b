"""The work that users of this library have it do, as cases that can be timed.

A case is a call (or the few calls that belong together) through the public entry points, at a size
that the repository's own configurations, tests and benchmark use or that lies between them:

* ``decode``   one decode step of attention of one layer over row caches
  (:meth:`cuda_ext.mixed_attn_decode`), from one short sequence to a batch of long ones and to a single
  sequence of a million tokens; optionally with the per-block softmax mass;
* ``paged``    the same over the block table of a ragged batch in one pool
  (:meth:`PagedLayerCache.attend`), the mass folded into its running mean;
* ``pack``     dense K/V of a prompt into packed row caches (:func:`pack_layout.pack_cache`);
* ``unpack``   a packed cache back into dense fp32 K/V (:func:`pack_layout.unpack_cache`);
* ``admit``    a batch of requests enters the pool: the slots of the batch before it are given back, the
  prompts are packed, demoted to their budget and attended once;
* ``chunks``   the maintenance loop: a prompt that arrives in chunks, demoted to the budget after each;
* ``chat``     admission of a small batch and its first decode steps, one token per sequence and step.

``listed()`` holds the cases that are always timed, ``draw`` gives more of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from geodesia_kv_b200.cuda_ext import get_ext
from geodesia_kv_b200.pack_layout import PackedCache, pack_cache, unpack_cache
from geodesia_kv_b200.paged import PagedLayerCache, PagedPool

BLOCK = 64
LADDER = (16, 8, 4, 2, 1)
# shares of the rungs 16, 8, 4, 2, centroid: the two mixes of the benchmark's workloads, the one the allocator
# leaves at 4 bits per value, and one rung alone
MIXES = {"warm": (0.10, 0.20, 0.40, 0.20, 0.10), "cold": (0.02, 0.08, 0.30, 0.40, 0.20), "budget4": (0.03, 0.09, 0.54, 0.0, 0.34),
         "bits8": (0.0, 1.0, 0.0, 0.0, 0.0), "bits4": (0.0, 0.0, 1.0, 0.0, 0.0), "bits2": (0.0, 0.0, 0.0, 1.0, 0.0)}
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DEV = "cuda"


def listed() -> list[dict]:
    return [
        # the first tokens of a chat: one short sequence, where latency and launches are what counts
        dict(name="decode_short", kind="decode", B=1, Hq=16, Hkv=2, D=128, group=32, T=1000, mix="warm", shared=False, mass=False),
        # one 16k-token sequence with a 3B-class head layout
        dict(name="decode_16k", kind="decode", B=1, Hq=16, Hkv=2, D=128, group=32, T=16384, mix="warm", shared=False, mass=False),
        # batched decode with an 8B-class head layout: the benchmark's main workload, one layer of it
        dict(name="decode_batch", kind="decode", B=32, Hq=32, Hkv=8, D=128, group=32, T=16384, mix="warm", shared=False, mass=False),
        # one sequence of a million tokens with a 7B-class head layout, mostly at the low rungs
        dict(name="decode_1m", kind="decode", B=1, Hq=28, Hkv=4, D=128, group=32, T=1048576, mix="cold", shared=False, mass=False),
        # head dim 64, one query head per cache row, the policy's default group, one rung vector for all rows
        dict(name="decode_d64", kind="decode", B=8, Hq=8, Hkv=8, D=64, group=16, T=3999, mix="warm", shared=True, mass=True),
        # serving: 256 sequences of lognormal length in one pool, demoted to 4 bits per value
        dict(name="paged_serving", kind="paged", B=256, Hq=16, Hkv=2, D=128, group=32, median=8192, longest=32768, budget=4.0, mass=True),
        # serving: a few sequences, no mass taken in this step
        dict(name="paged_few", kind="paged", B=6, Hq=32, Hkv=8, D=128, group=32, median=3000, longest=9000, budget=3.0, mass=False),
        # a batch of prompts of one layer into packed rows
        dict(name="pack_prompts", kind="pack", B=4, Hkv=8, D=128, group=32, T=16384, dtype="bf16", mix="warm"),
        # a cache handed back to a caller that wants dense K/V
        dict(name="unpack_rows", kind="unpack", B=2, Hkv=8, D=128, group=32, T=5000, dtype="fp16", mix="budget4"),
        # requests of different lengths enter the pool
        dict(name="admit_batch", kind="admit", B=8, Hq=32, Hkv=8, D=128, group=32, median=3000, longest=8192, budget=4.0, dtype="bf16"),
        # one long prompt per row in chunks of eight blocks
        dict(name="chunked_prompt", kind="chunks", B=4, Hq=32, Hkv=8, D=128, group=32, first=2048, chunk=512, steps=4, budget=4.0, dtype="bf16"),
        # a small batch from its prompts to its sixteenth token
        dict(name="chat_steps", kind="chat", B=3, Hq=16, Hkv=2, D=128, group=32, median=700, longest=1500, budget=4.0, steps=16, dtype="bf16"),
    ]


HEADS = ((16, 2), (32, 8), (28, 4), (8, 8), (7, 1), (8, 2), (32, 4))
SHAPES = ((128, 32), (128, 32), (128, 32), (128, 16), (128, 64), (64, 32), (64, 16), (64, 64))


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the ranges above (sizes over their logarithm, token counts of any remainder)."""
    kind = rng.choice(("decode", "decode", "decode", "paged", "paged", "pack", "pack", "unpack", "admit", "chunks", "chat"))
    Hq, Hkv = rng.choice(HEADS)
    D, group = rng.choice(SHAPES)
    c = dict(kind=kind, D=D, group=group)
    if kind == "decode":
        B = _log(rng, 1, 32)
        most = 4_000_000 // (B * Hkv)                                   # tokens per row: at most 4M in all rows
        c.update(B=B, Hq=Hq, Hkv=Hkv, T=_log(rng, 70, min(1048576, most)), mix=rng.choice(tuple(MIXES)), shared=rng.random() < 0.25,
                 mass=rng.random() < 0.3)
    elif kind == "paged":
        B = _log(rng, 1, 256)
        c.update(B=B, Hq=Hq, Hkv=Hkv, median=_log(rng, 200, max(400, min(8192, 3_000_000 // (B * Hkv)))), budget=round(rng.uniform(2.5, 8.0), 2),
                 mass=rng.random() < 0.7)
        c["longest"] = 4 * c["median"]
    elif kind in ("pack", "unpack"):
        B = _log(rng, 1, 8)
        c.update(B=B, Hkv=Hkv, T=_log(rng, 64, (524_288 if kind == "pack" else 200_000) // (B * Hkv)), dtype=rng.choice(("bf16", "bf16", "fp16", "fp32")),
                 mix=rng.choice(tuple(MIXES)))
    else:
        B = _log(rng, 1, 8)
        c.update(B=B, Hq=Hq, Hkv=Hkv, budget=round(rng.uniform(2.5, 8.0), 2), dtype=rng.choice(("bf16", "bf16", "fp16")))
        if kind == "chunks":
            n = rng.randint(1, 16)
            c.update(first=64 * rng.randint(1, 32), chunk=64 * n, steps=rng.randint(2, 5))
        else:
            c["median"] = _log(rng, 150, 3000)
            c["longest"] = 3 * c["median"]
            if kind == "chat":
                c["steps"] = rng.randint(4, 20)
    return c


# ---- inputs ------------------------------------------------------------------------------------------
def _lengths(case) -> np.ndarray:
    """Lengths of the sequences of a ragged batch: the quantiles of a lognormal (sigma 0.6) around the median, cut at the
    longest, in a fixed shuffled order.  Any remainder modulo the block size occurs."""
    B = case["B"]
    u = torch.special.ndtri((torch.arange(B, dtype=torch.float64) + 0.5) / B)
    n = np.rint(case["median"] * np.exp(0.6 * u.numpy())).astype(np.int64)
    return np.clip(n, 33, case["longest"])[np.random.default_rng(B).permutation(B)]


def _dense(gen, B, Hkv, T, D, dtype):
    """K with four outlier channels per head (x8), V ~ N(0, 1)."""
    k = torch.randn(B, Hkv, T, D, device=DEV, dtype=dtype, generator=gen)
    v = torch.randn(B, Hkv, T, D, device=DEV, dtype=dtype, generator=gen)
    ch = torch.rand(Hkv, D, device=DEV, generator=gen).argsort(-1)[:, :4]
    scale = torch.ones(Hkv, D, device=DEV, dtype=dtype).scatter_(1, ch, 8.0)
    k *= scale[None, :, None, :]
    return k, v


def _levels(gen, shape, mix):
    """Rungs of a mix in random order, the same number of each in every row; the first and the newest block stay
    exact (attention sink and open block)."""
    nb = shape[-1]
    edges = np.rint(np.cumsum((0.0,) + MIXES[mix]) * max(nb - 2, 0)).astype(np.int64)
    row = torch.from_numpy(np.repeat(np.array(LADDER, dtype=np.int32), np.diff(edges))).to(DEV)
    order = torch.rand(*shape[:-1], row.numel(), device=DEV, generator=gen).argsort(-1)
    level = torch.full(shape, 16, device=DEV, dtype=torch.int32)
    if nb > 2:
        level[..., 1:-1] = row[order]
    return level


def _query(gen, *shape):
    return torch.randn(*shape, device=DEV, generator=gen) * shape[-1] ** -0.5


def _mass(gen, lengths, Hkv, nb):
    """Running mass as attention leaves it: a power law of the distance from the newest block, a sink, some noise."""
    nblk = torch.from_numpy(np.repeat((lengths + BLOCK - 1) // BLOCK, Hkv)).to(DEV)[:, None]
    b = torch.arange(nb, device=DEV)[None]
    m = torch.where(b < nblk, (nblk - b).clamp_min(1).double() ** -1.2, torch.zeros((), device=DEV, dtype=torch.float64))
    m = m * torch.exp(0.5 * torch.randn(m.shape, device=DEV, generator=gen).double())
    m = m / m.sum(1, keepdim=True)
    m[:, 0] += 0.1
    return m.float()


def _pool(tokens_exact: int, Hkv: int, D: int, group: int) -> PagedPool:
    blocks = tokens_exact * Hkv // BLOCK + 64
    return PagedPool(int(blocks * 4 * BLOCK * D * 1.4) + (64 << 20), D, group, DEV)


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind, D, group = case["kind"], case["D"], case["group"]
    B, Hkv = case["B"], case["Hkv"]
    s = {"kind": kind, "case": case, "ext": get_ext()}
    if kind in ("decode", "pack", "unpack"):
        T = case["T"]
        nb = (T + BLOCK - 1) // BLOCK
        k, v = _dense(gen, B, Hkv, T, D, DTYPES[case.get("dtype", "bf16")])
        shared = case.get("shared", False)
        level = _levels(gen, (nb,) if shared else (B, Hkv, nb), case["mix"])
        if kind == "pack":
            s.update(k=k, v=v, level=level)
            return s
        cache = pack_cache(k, v, level, group)
        s["cache"] = cache
        if kind == "decode":
            s["q"] = _query(gen, B, case["Hq"], D)
            if shared:            # one metadata vector for every row, the reference's convention
                s["cache"] = PackedCache(cache.data, cache.offs[0, 0].contiguous(), cache.klo, cache.kstep, cache.vlo, cache.vstep,
                                         cache.level[0, 0].contiguous(), cache.valid[0, 0].contiguous(), group, D)
        return s
    Hq = case["Hq"]
    if kind == "chunks":
        total = case["first"] + case["chunk"] * case["steps"]
        lengths = np.full(B, total, dtype=np.int64)
    else:
        lengths = _lengths(case)
    T = int(lengths.max())
    steps = case.get("steps", 0) if kind == "chat" else 0
    k, v = _dense(gen, B, Hkv, T, D, DTYPES[case.get("dtype", "bf16")])
    nb = (T + steps + BLOCK - 1) // BLOCK
    pool = _pool(int(np.sum((lengths + BLOCK - 1) // BLOCK * BLOCK + BLOCK * 2)), Hkv, D, group)
    c = PagedLayerCache(pool, B, Hkv, cap_blocks=nb + 2)
    s.update(c=c, q=_query(gen, B, Hq, D), mass=_mass(gen, lengths, Hkv, nb + 2))
    if kind == "paged":
        c.prefill(k, v, lengths)
        c.maintain(case["budget"], mass=s["mass"][:, :c.nb])
        return s
    if kind == "chunks":
        f, n = case["first"], case["chunk"]
        cut = [0] + [f + i * n for i in range(case["steps"] + 1)]
        s["parts"] = [(k[:, :, a:b].contiguous(), v[:, :, a:b].contiguous()) for a, b in zip(cut[:-1], cut[1:])]
        return s
    s.update(k=k, v=v, lengths=lengths)
    if kind == "chat":
        s["qs"] = [_query(gen, B, Hq, D) for _ in range(steps)]
        s["new"] = [_dense(gen, B, Hkv, 1, D, k.dtype) for _ in range(steps)]
    return s


# ---- one pass -----------------------------------------------------------------------------------------
def run(s: dict):
    kind, case = s["kind"], s["case"]
    if kind == "decode":
        args = (s["q"], *s["cache"].kernel_args())
        return s["ext"].mixed_attn_decode_with_mass(*args) if case["mass"] else s["ext"].mixed_attn_decode(*args)
    if kind == "pack":
        p = pack_cache(s["k"], s["v"], s["level"], case["group"])
        return {"data": p.data, "offs": p.offs, "klo": p.klo, "kstep": p.kstep, "vlo": p.vlo, "vstep": p.vstep, "level": p.level, "valid": p.valid}
    if kind == "unpack":
        return unpack_cache(s["cache"])
    c = s["c"]
    if kind == "paged":
        if not case["mass"]:
            return c.attend(s["q"])
        out, mass = c.attend(s["q"], want_mass=True)
        c.observe(mass, 0.9)
        return out, mass
    c.release()                                   # the batch before this one leaves, its slots are used again
    if kind == "chunks":
        c.prefill(*s["parts"][0])
        c.maintain(case["budget"], mass=s["mass"][:, :c.nb])
        for k, v in s["parts"][1:]:
            c.extend(k, v)
            c.maintain(case["budget"], mass=s["mass"][:, :c.nb])
        return c.attend(s["q"], want_mass=True), c.level[:, :c.nb], c.valid[:, :c.nb], c.lens
    c.prefill(s["k"], s["v"], s["lengths"])
    c.maintain(case["budget"], mass=s["mass"][:, :c.nb])
    if kind == "admit":
        return c.attend(s["q"], want_mass=True), c.level[:, :c.nb], c.valid[:, :c.nb], c.lens
    outs = []
    for q, (k, v) in zip(s["qs"], s["new"]):
        c.append(k, v)
        out, mass = c.attend(q, want_mass=True)
        c.observe(mass, 0.9)
        outs.append(out)
    return outs, c.mass[:, :c.nb], c.level[:, :c.nb], c.valid[:, :c.nb], c.lens


# ---- what a pass cannot do without ----------------------------------------------------------------------
def _block_bytes(rung: int, D: int, group: int) -> int:
    data = 4 * D if rung == 1 else 4 * BLOCK * D if rung == 16 else BLOCK * D * rung // 4
    return data + (4 * (BLOCK // group * D + BLOCK * (D // group)) if rung in (8, 4, 2) else 0)


def _mix_bytes(case, nb: int) -> float:
    """Packed bytes of one row of nb blocks: the first and the last exact, the others of the mix."""
    exact = min(nb, 2)
    mean = sum(p * _block_bytes(r, case["D"], case["group"]) for p, r in zip(MIXES[case["mix"]], LADDER))
    return exact * _block_bytes(16, case["D"], case["group"]) + (nb - exact) * mean


def work(case: dict) -> dict:
    kind, D, B, Hkv = case["kind"], case["D"], case["B"], case["Hkv"]
    esize = {"bf16": 2, "fp16": 2, "fp32": 4}[case.get("dtype", "bf16")]
    if kind in ("decode", "pack", "unpack"):
        T = case["T"]
        nb = (T + BLOCK - 1) // BLOCK
        packed = B * Hkv * _mix_bytes(case, nb)
        meta = 16 * nb * (1 if case.get("shared") else B * Hkv)
        if kind == "pack":
            return {"bytes": packed + meta + 2 * B * Hkv * T * D * esize, "flops": 0.0}
        if kind == "unpack":
            return {"bytes": packed + meta + 2 * B * Hkv * nb * BLOCK * D * 4, "flops": 0.0}
        mass = 4 * B * Hkv * nb if case["mass"] else 0
        return {"bytes": packed + meta + mass + 8 * B * case["Hq"] * D, "flops": 4.0 * B * case["Hq"] * T * D}
    if kind == "chunks":
        tokens = B * (case["first"] + case["chunk"] * case["steps"])
    else:
        tokens = int(_lengths(case).sum())
    steps = case["steps"] if kind == "chat" else 1
    packed = tokens * Hkv * D * 2 * case["budget"] / 8
    read = steps * (packed + 8 * B * case["Hq"] * D)
    if kind != "paged":
        read += 2 * tokens * Hkv * D * esize + packed             # the dense rows once, the packed bytes written once
    return {"bytes": read, "flops": 4.0 * steps * tokens * case["Hq"] * D}


def tolerance(case: dict):
    """Packed bytes, scales and dequantised values are defined to the bit.  Attention outputs and masses are fp32 sums of
    products of exactly dequantised values, with the small operands carried as two 16-bit halves; the mean over a long
    sequence is small against its terms, so the error relative to it grows with the length.  Measured against attention in
    64 bits over 22 cases of these ranges: at most 2.9e-5 of the result's norm, 8.3e-5 of its root mean square at worst."""
    if case["kind"] in ("pack", "unpack"):
        return "exact"
    return {"rel": 1.2e-4, "max": 4e-4}
