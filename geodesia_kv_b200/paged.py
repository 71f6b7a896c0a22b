"""Paged packed KV cache: one byte pool per GPU, size-class free lists, per-row block tables.

The reference's serving plugin keeps one ``GeodesiaBlockCache`` per sequence in a dict
(``geodesia_kv/vllm_plugin/kv_cache.py:85-104``) and its capacity claim — more sequences per
GPU at a bit budget (``README.md:243-248``) — needs demotion to hand memory back.  Here it does:

* :class:`PagedPool` owns ONE ``uint8`` pool.  The pool is cut into slabs whose size is the least
  common multiple of the five slot sizes (1 474 560 bytes at D=128, g=32: 45 / 80 / 144 / 240 /
  2880 slots of the 16 / 8 / 4 / 2-bit / centroid rungs), so a slab serves exactly one rung with
  no waste and returns to the common free list when its last slot is freed.  A slot holds a block's
  bytes AND, for the quantised rungs, its four fp16 scale planes right behind them — a block is
  allocated, demoted ("allocate smaller, re-quantise, free larger") and freed as one piece.
* :class:`PagedLayerCache` is the block table of one layer: ``offs / level / valid`` of shape
  (sequences x KV heads, blocks), rows of different lengths padded with ``valid = 0``.  Prefill
  packs dense K/V straight into rung-16 slots, a decode step appends one token per row into the
  row's open block on the device, attention is ONE kernel call over the whole ragged batch (with
  the per-block softmax mass as a by-product), and maintenance runs the distortion, allocator and
  demotion kernels for all rows at once.

Free lists and block tables are mirrored on the host (native code over numpy arrays): a maintenance step reads the allocator's result back once,
for all rows (and, through :class:`PagedKVCache.maintain`, for all layers), which is the only
host synchronisation of the serving loop; decode steps in between launch kernels only.
"""
from __future__ import annotations

import ctypes as C
import math
import operator
import weakref
from typing import Sequence

import numpy as np
import torch

from . import _lib
from ._cuda import on, stream as _stream

BLOCK = 64
LADDER = (16, 8, 4, 2, 1)
_INDEX = {r: i for i, r in enumerate(LADDER)}
_DT = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}


def ladder_index_np(level: np.ndarray) -> np.ndarray:
    """Rungs (16, 8, 4, 2, 1) -> ladder indices 0..4."""
    lv = level.astype(np.int32)
    return (lv <= 8).astype(np.int32) + (lv <= 4) + (lv <= 2) + (lv <= 1)


_E_ARG, _E_POOL, _E_MEMORY = -6, -8, -9              # include/geodesia_kv_b200.h


def _addr(a: np.ndarray) -> int:
    return a.ctypes.data


def _lists(*sizes_and_types):
    """Host arrays side by side in one buffer, each from an 8-byte boundary: (buffer, arrays, their byte offsets)."""
    starts, end = [], 0
    for n, t in sizes_and_types:
        starts.append(end)
        end += (n * np.dtype(t).itemsize + 7) // 8 * 8
    buf = np.empty(end, dtype=np.uint8)
    return buf, [buf[at:at + n * np.dtype(t).itemsize].view(t) for (n, t), at in zip(sizes_and_types, starts)], starts


class PoolExhausted(RuntimeError):
    pass


class _Books:
    """The native bookkeeping of a pool (csrc/pool.cu) with the arrays that are its memory; the stacks of free slots are its
    own.  Shared by shallow copies of the pool; deep copies and pickles carry the state to a new one."""

    def __init__(self, slab_bytes: int, n_slabs: int, slot_bytes: Sequence[int]):
        self.args = (slab_bytes, n_slabs, tuple(slot_bytes))
        self.slab_rung = np.zeros(n_slabs, dtype=np.int32)           # 0 = unassigned
        self.slab_live = np.zeros(n_slabs, dtype=np.int64)
        self.free_slabs = np.empty(n_slabs, dtype=np.int64)
        self.counters = np.zeros(8, dtype=np.int64)      # free slabs, bytes in use, their peak, height of each rung's stack
        lib = _lib.load()
        self.handle = lib.gkv_pool_create(slab_bytes, n_slabs, (C.c_int64 * 5)(*slot_bytes), *map(_addr, self._arrays()))
        if not self.handle:
            raise MemoryError("no memory for the pool's bookkeeping")
        weakref.finalize(self, lib.gkv_pool_destroy, self.handle)

    def _arrays(self):
        return self.slab_rung, self.slab_live, self.free_slabs, self.counters

    def stacks(self) -> list:
        """Free slot offsets of every rung, the next one to hand out last (copies)."""
        lib = _lib.load()
        return [np.array((C.c_int64 * n).from_address(lib.gkv_pool_stack(self.handle, i)) if n else (), dtype=np.int64)
                for i, n in enumerate(self.counters[3:].tolist())]

    def __getstate__(self):
        return self.args, [a.copy() for a in self._arrays()], self.stacks()

    def __setstate__(self, state):
        args, arrays, stacks = state
        self.__init__(*args)
        for mine, a in zip(self._arrays(), arrays):
            mine[:] = a
        for i, s in enumerate(stacks):
            if _lib.load().gkv_pool_restore_stack(self.handle, i, s.size, _addr(s)):
                raise MemoryError("no memory for the pool's bookkeeping")


class PagedPool:
    """Byte pool with one free list per rung (host-side bookkeeping, device-side bytes)."""

    def __init__(self, capacity_bytes: int, D: int = 128, group: int = 32, device="cuda"):
        lib = _lib.load()
        self.D, self.group, self.device = D, group, torch.device(device)
        self.slot = {r: int(lib.gkv_paged_block_bytes(r, D, group)) for r in LADDER}
        if not all(self.slot.values()):
            raise ValueError(f"no paged layout for D={D}, group={group}")
        slab = 1
        for s in self.slot.values():
            slab = slab * s // math.gcd(slab, s)
        self.slab_bytes = slab if slab <= (8 << 20) else (2 << 20)
        self.n_slabs = int(capacity_bytes) // self.slab_bytes
        if self.n_slabs < 1:
            raise ValueError(f"capacity below one slab of {self.slab_bytes} bytes")
        self.data = torch.empty(self.n_slabs * self.slab_bytes, dtype=torch.uint8, device=self.device)
        self._books = _Books(self.slab_bytes, self.n_slabs, [self.slot[r] for r in LADDER])

    @property
    def lib(self):
        return _lib.load()

    @property
    def handle(self) -> int:
        return self._books.handle

    # -- accounting ---------------------------------------------------------------------------
    @property
    def _slab_rung(self) -> np.ndarray:
        return self._books.slab_rung

    @property
    def _slab_live(self) -> np.ndarray:
        return self._books.slab_live

    @property
    def _counters(self) -> np.ndarray:
        return self._books.counters

    @property
    def bytes_in_use(self) -> int:
        """Bytes of the slots handed out."""
        return int(self._counters[1])

    @bytes_in_use.setter
    def bytes_in_use(self, n: int) -> None:
        self._counters[1] = n

    @property
    def peak_bytes_in_use(self) -> int:
        """The most it has been; may be set, for instance back to ``bytes_in_use``."""
        return int(self._counters[2])

    @peak_bytes_in_use.setter
    def peak_bytes_in_use(self, n: int) -> None:
        self._counters[2] = n

    @property
    def _free_slabs(self) -> list:
        return self._books.free_slabs[:self._counters[0]].tolist()

    @property
    def _top(self) -> dict:
        return {r: int(self._counters[3 + i]) for i, r in enumerate(LADDER)}

    @property
    def _stack(self) -> dict:
        """Free slot offsets of every rung (a copy)."""
        return dict(zip(LADDER, self._books.stacks()))

    @property
    def capacity_bytes(self) -> int:
        return self.n_slabs * self.slab_bytes

    @property
    def bytes_reserved(self) -> int:
        """Bytes of the slabs that currently belong to a rung (slot granularity is bytes_in_use)."""
        return (self.n_slabs - int(self._counters[0])) * self.slab_bytes

    def slots_in_use(self, rung: int) -> int:
        return int(self._slab_live[self._slab_rung == rung].sum())

    # -- allocation ---------------------------------------------------------------------------
    def _check(self, rc: int, what: str) -> None:
        if rc == _E_POOL:
            raise PoolExhausted(f"pool of {self.capacity_bytes} bytes exhausted asking for {what} ({self.bytes_in_use} bytes in use)")
        if rc == _E_MEMORY:
            raise MemoryError("no memory for the pool's bookkeeping")
        if rc == _E_ARG:
            raise ValueError("an offset does not belong to a slab of its rung, or an entry lies beyond the table")
        _lib.check(rc, "pool")

    def alloc(self, rung: int, n: int) -> np.ndarray:
        """Offsets of n free slots of a rung (int64); refused with every slab where it was: smaller slots may still fit."""
        if n <= 0:
            return np.empty(0, dtype=np.int64)
        out = np.empty(operator.index(n), dtype=np.int64)
        self._check(self.lib.gkv_pool_alloc(self.handle, _INDEX[rung], out.size, _addr(out)), f"{n} slots of rung {rung}")
        return out

    def free(self, rung: int, offs: np.ndarray) -> None:
        """Give slots of a rung back; slabs left without a live slot return to the common list."""
        offs = np.ascontiguousarray(offs, dtype=np.int64)
        if offs.size:
            self._check(self.lib.gkv_pool_free(self.handle, _INDEX.get(rung, -1), offs.size, _addr(offs)), "a release")


class PagedLayerCache:
    """Block table of ONE layer over a :class:`PagedPool`: B sequences x Hkv heads, ragged lengths."""

    def __init__(self, pool: PagedPool, B: int, Hkv: int, cap_blocks: int = 64):
        self.pool, self.B, self.Hkv = pool, B, Hkv
        self.rows = B * Hkv
        self.D, self.group, self.device = pool.D, pool.group, pool.device
        self.lib = _lib.load()
        self.cap = 0
        self._bits = None
        self.len_h = np.zeros(B, dtype=np.int64)                     # tokens per sequence (host mirror)
        self.offs_h = np.full((self.rows, 0), -1, dtype=np.int64)
        self.level_h = np.zeros((self.rows, 0), dtype=np.int32)          # 0 = no block here
        self.offs = self.level = self.valid = self.mass = self.ek = self.ev = None
        self.lens = torch.zeros(self.rows, dtype=torch.int32, device=self.device)
        self.status = torch.zeros(1, dtype=torch.int32, device=self.device)
        self._grow(cap_blocks)

    # -- tables ---------------------------------------------------------------------------------
    def _grow(self, cap: int) -> None:
        dev, rows, old = self.device, self.rows, self.cap
        def wider(t, fill, dtype):
            new = torch.full((rows, cap), fill, dtype=dtype, device=dev)
            if t is not None and old:
                new[:, :old] = t
            return new
        self.offs = wider(self.offs, -1, torch.int64)
        self.level = wider(self.level, 0, torch.int32)
        self.valid = wider(self.valid, 0, torch.int32)
        self.mass = wider(self.mass, 0.0, torch.float32)
        self.ek = wider(self.ek, 0.0, torch.float32)
        self.ev = wider(self.ev, 0.0, torch.float32)
        oh = np.full((rows, cap), -1, dtype=np.int64)
        lh = np.zeros((rows, cap), dtype=np.int32)
        oh[:, :old], lh[:, :old] = self.offs_h, self.level_h
        self.offs_h, self.level_h, self.cap = oh, lh, cap

    @property
    def nb(self) -> int:
        """Blocks of the longest row (the width the kernels are called with)."""
        return int((int(self.len_h.max()) + BLOCK - 1) // BLOCK) if self.B else 0

    def blocks_per_seq(self) -> np.ndarray:
        return (self.len_h + BLOCK - 1) // BLOCK

    def _row_blocks(self) -> np.ndarray:
        return np.repeat(self.blocks_per_seq(), self.Hkv)

    def _upload(self, buf: np.ndarray, starts):
        """A buffer of host arrays -> (device buffer, the arrays' addresses in it), in ONE copy.  The caller holds the
        buffer until its kernel is launched; after that the stream order of the allocator protects it."""
        staged = torch.from_numpy(buf).to(self.device, non_blocking=True)
        base = staged.data_ptr()
        return staged, [base + at for at in starts]

    # -- growth ---------------------------------------------------------------------------------
    def prefill(self, k: torch.Tensor, v: torch.Tensor, lengths: Sequence[int] | None = None) -> None:
        """Pack the prompts: k, v (B, Hkv, T, D) dense; sequence b keeps its first lengths[b] tokens.

        Every block enters at rung 16 (exact bf16), as in the reference (policies.py:690-700)."""
        B, Hkv, T, D = k.shape
        if (B, Hkv, D) != (self.B, self.Hkv, self.D) or int(self.len_h.max(initial=0)) != 0:
            raise ValueError("prefill needs an empty cache of matching shape")
        k, v = k.contiguous(), v.contiguous()
        lengths = np.full(B, T, dtype=np.int64) if lengths is None else np.asarray(lengths, dtype=np.int64)
        if lengths.shape != (B,) or int(lengths.min()) < 1 or int(lengths.max()) > T:
            raise ValueError("one length per sequence, between 1 and the number of token rows given")
        nblk = (lengths + BLOCK - 1) // BLOCK
        if int(nblk.max()) + 1 > self.cap:
            self._grow(int(nblk.max()) + 1 + 16)
        self._enter(k, v, np.zeros(B, dtype=np.int64), nblk, T, lengths, fresh=False)
        self.len_h[:] = lengths

    def _enter(self, k, v, first: np.ndarray, count: np.ndarray, T: int, tokens, fresh: bool, len_add: int = 0, per_row: int = 0) -> None:
        """Give every sequence ``count`` blocks from block ``first`` on, at rung 16, in the slots reserved for them or new
        ones, and pack them: one upload, one kernel.  ``fresh`` clears the entries' mass and radii; the row lengths are set
        from ``tokens`` (valid tokens per sequence; None: whole blocks) or advanced by ``len_add`` (rows of ``per_row`` blocks)."""
        dev, n = self.device, int(count.sum()) * self.Hkv
        i64, i32 = np.int64, np.int32
        buf, (so, sl, at, nv, lv, *rl), starts = _lists((n, i64), (n, i64), (n, i64), (n, i32), (n, i32), *([(n, i32)] if tokens is not None else []))
        first, count = np.ascontiguousarray(first, dtype=i64), np.ascontiguousarray(count, dtype=i64)
        tokens = None if tokens is None else np.ascontiguousarray(tokens, dtype=i64)
        rc = self.lib.gkv_table_enter(self.pool.handle, _addr(self.offs_h), _addr(self.level_h), self.B, self.Hkv, self.cap, T, self.D,
                                      _addr(first), _addr(count), None if tokens is None else _addr(tokens), _addr(so), _addr(sl),
                                      _addr(at), _addr(nv), _addr(lv), _addr(rl[0]) if rl else None)
        self.pool._check(rc, f"the slots of {n} blocks")
        with on(dev):
            staged, (src, dst, at, nv, lv, *rl) = self._upload(buf, starts)
            rc = self.lib.gkv_paged_enter_blocks(k.data_ptr(), v.data_ptr(), _DT[k.dtype], src, int(self.D), nv,
                                                 self.pool.data.data_ptr(), dst, lv, at, self.offs.data_ptr(),
                                                 self.level.data_ptr(), self.valid.data_ptr(),
                                                 self.mass.data_ptr() if fresh else None, self.ek.data_ptr() if fresh else None,
                                                 self.ev.data_ptr() if fresh else None, self.lens.data_ptr(), rl[0] if rl else None,
                                                 len_add, per_row, self.cap, n, self.D, BLOCK, self.group, _stream(dev))
        _lib.check(rc, "gkv_paged_enter_blocks")

    def extend(self, k: torch.Tensor, v: torch.Tensor) -> None:
        """Append whole blocks to EVERY sequence: k, v (B, Hkv, n*64, D) dense; all sequences must
        stand at a block boundary (chunked prefill, or a serving loop that packs a block at a time)."""
        B, Hkv, T, D = k.shape
        if (B, Hkv, D) != (self.B, self.Hkv, self.D) or T % BLOCK or np.any(self.len_h % BLOCK):
            raise ValueError("extend appends whole blocks to sequences that stand at a block boundary")
        k, v = k.contiguous(), v.contiguous()
        n = T // BLOCK
        first = self.len_h // BLOCK
        if int(first.max()) + n + 1 > self.cap:
            self._grow(int(first.max()) + n + 1 + 63)
        self._enter(k, v, first, np.full(B, n, dtype=np.int64), T, None, fresh=True, len_add=T, per_row=n)
        self.len_h += T

    def pack_blocks(self, k, v, src_off, token_stride, nvalid, slots, levels, radii: bool = False):
        """Quantise blocks from dense rows into given slots (element offsets into k and v)."""
        dev = self.device
        n = int(len(slots))
        up = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(dev, non_blocking=True).to(dt)
        so, nv, sl, lv = up(src_off, torch.int64), up(nvalid, torch.int32), up(slots, torch.int64), up(levels, torch.int32)
        ek = torch.zeros(n, dtype=torch.float32, device=dev) if radii else None
        ev = torch.zeros(n, dtype=torch.float32, device=dev) if radii else None
        with on(dev):
            rc = self.lib.gkv_paged_pack_blocks(k.data_ptr(), v.data_ptr(), _DT[k.dtype], so.data_ptr(), int(token_stride),
                                                nv.data_ptr(), self.pool.data.data_ptr(), sl.data_ptr(), lv.data_ptr(),
                                                ek.data_ptr() if radii else None, ev.data_ptr() if radii else None,
                                                n, self.D, BLOCK, self.group, _stream(dev))
        _lib.check(rc, "gkv_paged_pack_blocks")
        return ek, ev

    def append(self, k_new: torch.Tensor, v_new: torch.Tensor) -> None:
        """One more token for every sequence: k_new, v_new (B, Hkv, 1, D) or (B, Hkv, D)."""
        if (self.len_h % BLOCK == 0).any():                               # some sequence opens a new block
            self.reserve(1)
        self.append_device(k_new, v_new)
        self.len_h += 1

    def reserve(self, tokens: int) -> None:
        """Give every row the rung-16 slots its next ``tokens`` appended tokens will need, so that that
        many :meth:`append_device` calls (e.g. replays of a captured step) need no host work."""
        first = (self.len_h + BLOCK - 1) // BLOCK                       # first block without a slot yet
        last = (self.len_h + tokens + BLOCK - 1) // BLOCK               # one past the last block needed
        cnt = np.maximum(last - first, 0)
        if int(cnt.sum()) == 0:
            return
        if int(last.max()) + 1 > self.cap:
            self._grow(int(last.max()) + 1 + 63)
        seq = np.repeat(np.arange(self.B), cnt)
        blk = np.arange(int(cnt.sum())) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(first, cnt)
        rows = (seq[:, None] * self.Hkv + np.arange(self.Hkv)[None]).reshape(-1)
        blks = np.repeat(blk, self.Hkv)
        have = self.offs_h[rows, blks] >= 0
        rows, blks = rows[~have], blks[~have]
        slots = self.pool.alloc(16, rows.size)
        self.offs_h[rows, blks] = slots
        self.level_h[rows, blks] = 16
        flat, dev = rows * self.cap + blks, self.device
        with on(dev):
            buf, (a, b), starts = _lists((flat.size, np.int64), (slots.size, np.int64))
            a[:], b[:] = flat, slots
            staged, (at, so) = self._upload(buf, starts)
            rc = self.lib.gkv_paged_open_blocks(at, so, int(flat.size), self.offs.data_ptr(), self.level.data_ptr(),
                                                self.mass.data_ptr(), self.ek.data_ptr(), self.ev.data_ptr(), _stream(dev))
        _lib.check(rc, "gkv_paged_open_blocks")

    def sync_lengths(self) -> None:
        """Re-read the row lengths from the device (after append_device calls the host did not count)."""
        self.len_h[:] = self.lens.cpu().numpy().reshape(self.B, self.Hkv)[:, 0]

    def append_device(self, k_new: torch.Tensor, v_new: torch.Tensor) -> None:
        """The device half of :meth:`append` (no host bookkeeping): safe inside a CUDA graph as long
        as no row crosses into a block without a slot — the status word says if one did."""
        n = self.rows * self.D
        if not (k_new.numel() == v_new.numel() == n and k_new.is_contiguous() and v_new.is_contiguous()):
            k_new, v_new = k_new.reshape(self.rows, self.D).contiguous(), v_new.reshape(self.rows, self.D).contiguous()
        dev = self.device
        with on(dev):
            rc = self.lib.gkv_paged_append_token(k_new.data_ptr(), v_new.data_ptr(), _DT[k_new.dtype],
                                                 self.pool.data.data_ptr(), self.offs.data_ptr(), self.valid.data_ptr(),
                                                 self.lens.data_ptr(), self.status.data_ptr(), self.rows, self.cap,
                                                 self.D, BLOCK, _stream(dev))
        _lib.check(rc, "gkv_paged_append_token")

    # -- attention ------------------------------------------------------------------------------
    def attend(self, q: torch.Tensor, want_mass: bool = False, nb: int | None = None):
        """q (B, Hq, D) float32, already scaled -> out (B, Hq, D) [, mass (rows, table width)]: one kernel call."""
        from .cuda_ext import get_ext
        ext = get_ext()
        B, Hq, D = q.shape
        if B != self.B or D != self.D or q.dtype != torch.float32 or not q.is_contiguous():
            raise RuntimeError("q must be contiguous float32 (B, Hq, D) matching the cache")
        # by default the whole table goes in: entries beyond a row's blocks have valid = 0 and are never read
        nb = self.cap if nb is None else nb
        dev = self.device
        offs, level, valid = self.offs, self.level, self.valid
        if nb != self.cap:                                           # the kernel wants tables of width nb
            offs, level, valid = offs[:, :nb].contiguous(), level[:, :nb].contiguous(), valid[:, :nb].contiguous()
        lib = self.lib
        with on(dev):
            need = (lib.gkv_decode_mass_workspace_bytes(B, Hq, self.Hkv, D, nb, self.group) if want_mass
                    else lib.gkv_decode_workspace_bytes(B, Hq, self.Hkv, D, nb))
            ws = ext._workspace(dev, need)
            out = torch.empty(B, Hq, D, dtype=torch.float32, device=dev)
            mass = torch.empty(self.rows, nb, dtype=torch.float32, device=dev) if want_mass else None
            rc = lib.gkv_paged_attn_decode(q.data_ptr(), self.pool.data.data_ptr(), self.pool.data.numel(), offs.data_ptr(),
                                           level.data_ptr(), valid.data_ptr(), out.data_ptr(),
                                           mass.data_ptr() if want_mass else None, None, ws.data_ptr(), ws.numel(),
                                           B, Hq, self.Hkv, D, nb, BLOCK, self.group, _stream(dev))
        _lib.check(rc, "gkv_paged_attn_decode")
        return (out, mass) if want_mass else out

    def observe(self, mass: torch.Tensor, decay: float) -> None:
        """Fold one step's per-block mass (rows, nb) into the running mass (policies.py:705-708)."""
        nb = mass.shape[1]
        (self.mass if nb == self.cap else self.mass[:, :nb]).lerp_(mass, 1.0 - decay)

    # -- maintenance ----------------------------------------------------------------------------
    def hot_blocks(self, nb: int, sinks: int = 4, window: int = 128) -> torch.Tensor:
        """(rows, nb) uint8: blocks that must stay exact — sinks, the recent window, the block being
        written and its predecessor (policies.py:677-681), per row of the ragged batch."""
        lens = self.lens.to(torch.int64)[:, None]
        b = torch.arange(nb, device=self.device)[None]
        nbr = (lens + BLOCK - 1) // BLOCK
        hot = (b < max(1, (sinks + BLOCK - 1) // BLOCK)) | (b >= (lens - 1) // BLOCK - 1) | \
              (b >= nbr - max(1, (window + BLOCK - 1) // BLOCK))
        return (hot & (b < nbr)).to(torch.uint8).contiguous()

    def _ladder_bits(self):
        """Bits of a block at each rung, as the library takes them."""
        if self._bits is None:
            from .policies import ladder_bits
            self._bits = (C.c_float * 5)(*ladder_bits(BLOCK, self.D, self.group))
        return self._bits

    def plan_demotion(self, budget_bits: float, sinks: int = 4, window: int = 128, mass_power: float = 1.0,
                      value_weight: float = 0.0, mass: torch.Tensor | None = None) -> torch.Tensor:
        """Run the distortion and allocator kernels over every row; returns the target ladder index
        (rows, nb) int32 ON THE DEVICE (nothing is read back here).  ``mass``: (rows, nb) or wider, any shape of
        rows * nb values in that order (the (B, Hkv, nb) of the decode calls), or what broadcasts to (rows, nb)."""
        nb, dev, rows, D = self.nb, self.device, self.rows, self.D
        m = self.mass if mass is None else mass
        shape = m.shape
        if len(shape) != 2 or shape[0] != rows:
            m = m.reshape(rows, nb) if m.numel() == rows * nb else m.expand(rows, nb)
            shape = m.shape
        apart, step = m.stride()
        if m.dtype != torch.float32 or step != 1 or apart < nb or shape[1] < nb:
            m = (m[:, :nb] if shape[1] > nb else m.expand(rows, nb)).to(torch.float32).contiguous()
            apart = nb                               # a single row may have any stride
        E = torch.empty(rows, nb, 5, dtype=torch.float32, device=dev)
        tgt = torch.empty(rows, nb, dtype=torch.int32, device=dev)
        bits = self._ladder_bits()
        need = self.lib.gkv_paged_plan_ratio_bytes(bits, rows, nb)
        ratio = torch.empty(need, dtype=torch.uint8, device=dev) if need else None
        with on(dev):
            rc = self.lib.gkv_paged_plan_demotion(self.pool.data.data_ptr(), self.offs.data_ptr(), self.level.data_ptr(),
                                                  self.lens.data_ptr(), m.data_ptr(), apart, bits,
                                                  float(budget_bits * 2.0 * BLOCK * D), max(1, (sinks + BLOCK - 1) // BLOCK),
                                                  max(1, (window + BLOCK - 1) // BLOCK), float(mass_power), float(value_weight),
                                                  E.data_ptr(), ratio.data_ptr() if need else None, tgt.data_ptr(), rows, nb,
                                                  self.cap, D, BLOCK, self.group, _stream(dev))
        _lib.check(rc, "gkv_paged_plan_demotion")
        return tgt

    def apply_demotion(self, tgt_idx_host: np.ndarray) -> int:
        """Demote to the allocator's result (host array (rows, nb) of ladder indices): allocate the
        smaller slots, re-quantise on the device, free the larger slots.  Returns blocks demoted."""
        nb, lib, dev = tgt_idx_host.shape[1], self.lib, self.device
        if nb > self.cap:
            raise ValueError(f"targets for {nb} blocks, the table has {self.cap}")
        if tgt_idx_host.dtype != np.int32:
            if tgt_idx_host.dtype.kind not in "iub":
                raise IndexError("targets are ladder indices, which are integers")
            tgt_idx_host = np.clip(tgt_idx_host, 0, 4)                # whatever is out of range stays so in 32 bits
        tgt = np.ascontiguousarray(np.broadcast_to(tgt_idx_host, (self.rows, nb)), dtype=np.int32)
        blocks = self.blocks_per_seq()
        table = (_addr(self.offs_h), _addr(self.level_h), self.B, self.Hkv, self.cap, _addr(blocks), _addr(tgt), nb)
        n = int(lib.gkv_table_demotions(*table))
        if n == 0:
            return 0
        i64, i32 = np.int64, np.int32
        buf, lists, starts = _lists((n, i64), (n, i64), (n, i64), (n, i32), (n, i32))
        old, new, at, lo, ln = map(_addr, lists)
        self.pool._check(lib.gkv_table_plan_demotion(self.pool.handle, *table, n, old, new, at, lo, ln), f"the slots of {n} demoted blocks")
        with on(dev):
            staged, (d_old, d_new, d_at, d_lo, d_ln) = self._upload(buf, starts)
            rc = lib.gkv_paged_demote_entries(self.pool.data.data_ptr(), d_old, d_lo, d_new, d_ln, d_at, self.offs.data_ptr(),
                                              self.level.data_ptr(), self.ek.data_ptr(), self.ev.data_ptr(), n, self.D,
                                              BLOCK, self.group, _stream(dev))
        _lib.check(rc, "gkv_paged_demote_entries")
        # the old slots are free for whatever is launched after the demotion kernel on this stream
        self.pool._check(lib.gkv_table_apply_demotion(self.pool.handle, *table[:2], n, old, new, at, lo, ln), "a release")
        return n

    def maintain(self, budget_bits: float, **kw) -> int:
        """plan_demotion + one read-back + apply_demotion for this layer alone."""
        if budget_bits <= 0 or self.nb == 0:
            return 0
        return self.apply_demotion(self.plan_demotion(budget_bits, **kw).cpu().numpy())

    # -- accounting / debugging -----------------------------------------------------------------
    def bytes_in_pool(self) -> int:
        used = np.arange(self.cap)[None, :] < self._row_blocks()[:, None]
        lv = self.level_h[used]
        return int(sum(int((lv == r).sum()) * self.pool.slot[r] for r in LADDER))

    def bits_per_value(self) -> float:
        """Resident bits per cached value with the reference's accounting (policies.py:1582-1596)."""
        from .policies import ladder_bits
        used = np.arange(self.cap)[None, :] < self._row_blocks()[:, None]
        bits = np.array(ladder_bits(BLOCK, self.D, self.group))[ladder_index_np(self.level_h[used])]
        return float(bits.sum()) / max(1, int(used.sum()) * 2 * BLOCK * self.D)

    def release(self) -> None:
        """Give every slot back to the pool, also those that :meth:`reserve` opened and no token has reached."""
        self.pool._check(self.lib.gkv_table_release(self.pool.handle, _addr(self.offs_h), _addr(self.level_h), self.offs_h.size), "a release")
        self.len_h[:] = 0
        dev = self.device
        with on(dev):
            rc = self.lib.gkv_paged_clear_table(self.offs.data_ptr(), self.level.data_ptr(), self.valid.data_ptr(),
                                                self.mass.data_ptr(), self.ek.data_ptr(), self.ev.data_ptr(), self.lens.data_ptr(),
                                                self.rows, self.cap, _stream(dev))
        _lib.check(rc, "gkv_paged_clear_table")

    def dequantise(self):
        """Exact fp32 K, V (rows, nb*64, D) of the cached tokens (tests, debugging); padding is zero."""
        nb, dev = self.nb, self.device
        k = torch.zeros(self.rows, nb, BLOCK, self.D, dtype=torch.float32, device=dev)
        v = torch.zeros_like(k)
        offs, level = self.offs[:, :nb].contiguous(), self.level[:, :nb].contiguous()
        with on(dev):
            rc = self.lib.gkv_paged_unpack_blocks(self.pool.data.data_ptr(), offs.data_ptr(), level.data_ptr(),
                                                  k.data_ptr(), v.data_ptr(), self.rows * nb, self.D, BLOCK, self.group,
                                                  _stream(dev))
        _lib.check(rc, "gkv_paged_unpack_blocks")
        return k.view(self.rows, nb * BLOCK, self.D), v.view(self.rows, nb * BLOCK, self.D)
