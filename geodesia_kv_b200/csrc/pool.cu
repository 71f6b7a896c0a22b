// Host-side bookkeeping of the block pool and of a layer's block table: which slots are free, which slot a block gets, which
// entries a demotion changes.  No kernels.
//
// A maintenance step moves a few thousand slots, and everything here happens between two launches that wait for it: numpy
// needed 20 to 40 us per operation for passes over small arrays (masks, gathers, a histogram per rung), six of them per step
// and ten per admission.  One pass in C over the table takes one or two microseconds per thousand blocks.
//
// Nothing here throws, and a request that is refused for lack of slots leaves everything as it was.  The caller serialises
// calls on one pool (the Python face holds the interpreter lock across them).  8 requests of a batch admitted 883 -> 509 us, a
// prompt in five chunks 1712 -> 1067.
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <new>

#include "gkv_common.cuh"

namespace gkv {

constexpr int kRungs = 5;      // ladder indices 0..4: rungs 16, 8, 4, 2, centroid

struct Pool {
    int64_t slab_bytes, n_slabs, slot[kRungs];
    double per_byte;           // 1 / slab_bytes
    // shared with the caller, who allocated them: slab -> rung (0 = unassigned), live slots of a slab, stack of free slabs,
    // counters (free slabs, bytes in use, their peak, then the height of each rung's stack)
    int32_t* slab_rung;
    int64_t* slab_live;
    int64_t* free_slabs;
    int64_t* n;
    int64_t* stack[kRungs];    // free slots of every rung, the next one to hand out on top
    int64_t room[kRungs];
    int64_t* emptied;          // slabs that a free leaves without a live slot
    int64_t emptied_room;
};
enum { kFreeSlabs = 0, kBytes = 1, kPeak = 2, kTop = 3 };

// Slab of an offset of the pool.  A 64-bit division here was most of what a release costs (3400 blocks of five rungs: 86 us
// with it, 52 without).
static inline int64_t slab_of(const Pool& p, int64_t off) {
    const int64_t s = (int64_t)((double)off * p.per_byte);       // off by one at most
    return off < s * p.slab_bytes ? s - 1 : off >= (s + 1) * p.slab_bytes ? s + 1 : s;
}

static bool grow(int64_t*& a, int64_t& room, int64_t need) {
    if (need <= room) return true;
    const int64_t to = std::max<int64_t>(std::max<int64_t>(2 * room, need), 1024);
    int64_t* p = static_cast<int64_t*>(realloc(a, (size_t)to * sizeof(int64_t)));
    if (!p) return false;
    a = p;
    room = to;
    return true;
}

// Slabs that n slots of a rung take from the common list.
static int64_t slabs_for(const Pool& p, int r, int64_t n) {
    const int64_t per_slab = p.slab_bytes / p.slot[r], top = p.n[kTop + r];
    return n > top ? (n - top + per_slab - 1) / per_slab : 0;
}

// Everything that can refuse slots of all rungs together, before any is handed out.
static int check_alloc(Pool& p, const int64_t (&n)[kRungs]) {
    int64_t need = 0;
    for (int r = 0; r < kRungs; ++r) need += slabs_for(p, r, n[r]);
    if (need > p.n[kFreeSlabs]) return GKV_E_POOL;
    for (int r = 0; r < kRungs; ++r)
        if (!grow(p.stack[r], p.room[r], p.n[kTop + r] + slabs_for(p, r, n[r]) * (p.slab_bytes / p.slot[r]))) return GKV_E_MEMORY;
    return GKV_OK;
}

static void do_alloc(Pool& p, int r, int64_t n, int64_t* out) {
    const int64_t size = p.slot[r], per_slab = p.slab_bytes / size, need = slabs_for(p, r, n);
    int64_t& top = p.n[kTop + r];
    for (int64_t i = 0; i < need; ++i) {
        const int64_t s = p.free_slabs[--p.n[kFreeSlabs]];
        p.slab_rung[s] = ladder_level(r);
        // pushed high to low, so low addresses are handed out first
        for (int64_t k = per_slab - 1; k >= 0; --k) p.stack[r][top++] = s * p.slab_bytes + k * size;
    }
    for (int64_t i = 0; i < n; ++i) {
        out[i] = p.stack[r][--top];
        ++p.slab_live[slab_of(p, out[i])];
    }
    p.n[kBytes] += n * size;
    p.n[kPeak] = std::max(p.n[kPeak], p.n[kBytes]);
}

static int pool_alloc(Pool& p, int r, int64_t n, int64_t* out) {
    if (n <= 0) return GKV_OK;
    int64_t want[kRungs] = {0};
    want[r] = n;
    if (const int rc = check_alloc(p, want)) return rc;
    do_alloc(p, r, n, out);
    return GKV_OK;
}

// Everything that can refuse a release, before anything of it is done.
static int check_free(Pool& p, int r, int64_t n, const int64_t* offs) {
    const int32_t rung = ladder_level(r);
    for (int64_t i = 0; i < n; ++i) {
        if (offs[i] < 0 || offs[i] >= p.n_slabs * p.slab_bytes || p.slab_rung[slab_of(p, offs[i])] != rung) return GKV_E_ARG;
    }
    return grow(p.stack[r], p.room[r], p.n[kTop + r] + n) && grow(p.emptied, p.emptied_room, std::min(n, p.n_slabs)) ? GKV_OK : GKV_E_MEMORY;
}

static void do_free(Pool& p, int r, int64_t n, const int64_t* offs) {
    const int32_t rung = ladder_level(r);
    int64_t& top = p.n[kTop + r];
    for (int64_t i = 0; i < n; ++i) {
        p.stack[r][top++] = offs[i];
        --p.slab_live[slab_of(p, offs[i])];
    }
    p.n[kBytes] -= n * p.slot[r];
    int64_t m = 0;
    for (int64_t i = 0; i < n; ++i) {
        const int64_t s = slab_of(p, offs[i]);
        if (p.slab_live[s] == 0 && p.slab_rung[s] == rung) {
            p.slab_rung[s] = 0;                          // once per slab
            p.emptied[m++] = s;
        }
    }
    if (m) {
        int64_t keep = 0;                                // the stack's other slots are of slabs in use
        for (int64_t i = 0; i < top; ++i)
            if (p.slab_rung[slab_of(p, p.stack[r][i])] == rung) p.stack[r][keep++] = p.stack[r][i];
        top = keep;
        std::sort(p.emptied, p.emptied + m);
        for (int64_t i = m - 1; i >= 0; --i) p.free_slabs[p.n[kFreeSlabs]++] = p.emptied[i];
    }
}

static int pool_free(Pool& p, int r, int64_t n, const int64_t* offs) {
    if (n <= 0) return GKV_OK;
    if (const int rc = check_free(p, r, n, offs)) return rc;
    do_free(p, r, n, offs);
    return GKV_OK;
}

// Offsets of `n` entries sorted by rung (each rung's in order): start[r] .. start[r + 1] of `out`.
static void by_rung(const int64_t* offs, const int32_t* level, int64_t n, int64_t* out, int64_t (&start)[kRungs + 1]) {
    int64_t cnt[kRungs] = {0};
    for (int64_t i = 0; i < n; ++i)
        if (offs[i] >= 0 && level_ok(level[i])) ++cnt[ladder_index(level[i])];
    start[0] = 0;
    for (int r = 0; r < kRungs; ++r) start[r + 1] = start[r] + cnt[r];
    int64_t at[kRungs];
    for (int r = 0; r < kRungs; ++r) at[r] = start[r];
    for (int64_t i = 0; i < n; ++i)
        if (offs[i] >= 0 && level_ok(level[i])) out[at[ladder_index(level[i])]++] = offs[i];
}

static int free_by_rung(Pool& p, const int64_t* offs, const int32_t* level, int64_t n) {
    if (n <= 0) return GKV_OK;
    int64_t* sorted = static_cast<int64_t*>(malloc((size_t)n * sizeof(int64_t)));
    if (!sorted) return GKV_E_MEMORY;
    int64_t start[kRungs + 1];
    by_rung(offs, level, n, sorted, start);
    int rc = GKV_OK;
    for (int r = 0; r < kRungs && rc == GKV_OK; ++r) rc = check_free(p, r, start[r + 1] - start[r], sorted + start[r]);
    for (int r = 0; r < kRungs && rc == GKV_OK; ++r) do_free(p, r, start[r + 1] - start[r], sorted + start[r]);
    free(sorted);
    return rc;
}

// Does the block change, and to which ladder index?
static inline bool demoted(int32_t tgt, int32_t level, int64_t off, int& idx) {
    idx = tgt < 0 ? 0 : tgt > kRungs - 1 ? kRungs - 1 : tgt;
    return off >= 0 && ladder_level(idx) < level;
}

}  // namespace gkv

extern "C" {

void* gkv_pool_create(int64_t slab_bytes, int64_t n_slabs, const int64_t* slot_bytes, int32_t* slab_rung, int64_t* slab_live,
                      int64_t* free_slabs, int64_t* counters) {
    if (slab_bytes <= 0 || n_slabs <= 0 || !slot_bytes || !slab_rung || !slab_live || !free_slabs || !counters) return nullptr;
    gkv::Pool* p = new (std::nothrow) gkv::Pool();
    if (!p) return nullptr;
    p->slab_bytes = slab_bytes; p->n_slabs = n_slabs; p->per_byte = 1.0 / (double)slab_bytes;
    for (int r = 0; r < gkv::kRungs; ++r) {
        if (slot_bytes[r] <= 0 || slot_bytes[r] > slab_bytes) { delete p; return nullptr; }
        p->slot[r] = slot_bytes[r];
    }
    p->slab_rung = slab_rung; p->slab_live = slab_live; p->free_slabs = free_slabs; p->n = counters;
    for (int64_t s = 0; s < n_slabs; ++s) free_slabs[s] = n_slabs - 1 - s;
    memset(counters, 0, (gkv::kTop + gkv::kRungs) * sizeof(int64_t));
    counters[gkv::kFreeSlabs] = n_slabs;
    return p;
}

void gkv_pool_destroy(void* pool) {
    gkv::Pool* p = static_cast<gkv::Pool*>(pool);
    if (!p) return;
    for (int r = 0; r < gkv::kRungs; ++r) free(p->stack[r]);
    free(p->emptied);
    delete p;
}

const int64_t* gkv_pool_stack(void* pool, int rung_index) {
    return pool && rung_index >= 0 && rung_index < gkv::kRungs ? static_cast<gkv::Pool*>(pool)->stack[rung_index] : nullptr;
}

int gkv_pool_restore_stack(void* pool, int rung_index, int64_t n, const int64_t* slots) {
    if (!pool || (n > 0 && !slots)) return GKV_E_NULL;
    if (rung_index < 0 || rung_index >= gkv::kRungs || n < 0) return GKV_E_ARG;
    gkv::Pool& p = *static_cast<gkv::Pool*>(pool);
    if (!gkv::grow(p.stack[rung_index], p.room[rung_index], n)) return GKV_E_MEMORY;
    if (n > 0) memcpy(p.stack[rung_index], slots, (size_t)n * sizeof(int64_t));
    p.n[gkv::kTop + rung_index] = n;
    return GKV_OK;
}

int gkv_pool_alloc(void* pool, int rung_index, int64_t n, int64_t* out) {
    if (!pool || (n > 0 && !out)) return GKV_E_NULL;
    if (rung_index < 0 || rung_index >= gkv::kRungs) return GKV_E_ARG;
    return gkv::pool_alloc(*static_cast<gkv::Pool*>(pool), rung_index, n, out);
}

int gkv_pool_free(void* pool, int rung_index, int64_t n, const int64_t* offs) {
    if (!pool || (n > 0 && !offs)) return GKV_E_NULL;
    if (rung_index < 0 || rung_index >= gkv::kRungs) return GKV_E_ARG;
    return gkv::pool_free(*static_cast<gkv::Pool*>(pool), rung_index, n, offs);
}

int gkv_table_release(void* pool, int64_t* offs, int32_t* level, int64_t entries) {
    if (!pool || !offs || !level) return GKV_E_NULL;
    const int rc = gkv::free_by_rung(*static_cast<gkv::Pool*>(pool), offs, level, entries);
    if (rc) return rc;
    for (int64_t i = 0; i < entries; ++i) { offs[i] = -1; level[i] = 0; }
    return GKV_OK;
}

int gkv_table_enter(void* pool, int64_t* offs, int32_t* level, int B, int Hkv, int cap, int64_t T, int D, const int64_t* first,
                    const int64_t* count, const int64_t* tokens, int64_t* src_off, int64_t* slots, int64_t* flat, int32_t* nvalid,
                    int32_t* rung, int32_t* row_len) {
    if (!pool || !offs || !level || !first || !count || !src_off || !slots || !flat || !nvalid || !rung) return GKV_E_NULL;
    int64_t fresh = 0, total = 0;
    for (int b = 0; b < B; ++b) {
        if (first[b] < 0 || count[b] < 0 || first[b] + count[b] > cap) return GKV_E_ARG;
        for (int h = 0; h < Hkv; ++h)
            for (int64_t i = 0; i < count[b]; ++i) fresh += offs[((int64_t)b * Hkv + h) * cap + first[b] + i] < 0;
        total += count[b] * Hkv;
    }
    // the new slots wait at the end of the list of all
    int64_t* got = slots + (total - fresh);
    if (const int rc = gkv::pool_alloc(*static_cast<gkv::Pool*>(pool), 0, fresh, got)) return rc;
    int64_t k = 0;
    for (int b = 0; b < B; ++b)
        for (int h = 0; h < Hkv; ++h) {
            const int64_t row = (int64_t)b * Hkv + h;
            for (int64_t i = 0; i < count[b]; ++i, ++k) {
                const int64_t at = row * cap + first[b] + i;
                slots[k] = offs[at] < 0 ? *got++ : offs[at];      // slots reserved earlier are used first
                offs[at] = slots[k];
                level[at] = 16;
                src_off[k] = (row * T + i * gkv::kP) * D;
                flat[k] = at;
                const int64_t left = tokens ? tokens[b] - i * gkv::kP : gkv::kP;
                nvalid[k] = (int32_t)std::min<int64_t>(gkv::kP, left);
                rung[k] = 16;
                if (row_len) row_len[k] = tokens ? (int32_t)tokens[b] : 0;
            }
        }
    return GKV_OK;
}

int64_t gkv_table_demotions(const int64_t* offs, const int32_t* level, int B, int Hkv, int cap, const int64_t* blocks,
                            const int32_t* tgt, int nb) {
    if (!offs || !level || !blocks || !tgt) return 0;
    int64_t n = 0;
    for (int64_t row = 0; row < (int64_t)B * Hkv; ++row) {
        const int64_t used = std::min<int64_t>(blocks[row / Hkv], std::min(nb, cap));
        int idx;
        for (int64_t b = 0; b < used; ++b) n += gkv::demoted(tgt[row * nb + b], level[row * cap + b], offs[row * cap + b], idx);
    }
    return n;
}

int gkv_table_plan_demotion(void* pool, const int64_t* offs, const int32_t* level, int B, int Hkv, int cap, const int64_t* blocks,
                            const int32_t* tgt, int nb, int64_t n, int64_t* off_old, int64_t* off_new, int64_t* flat,
                            int32_t* level_old, int32_t* level_new) {
    if (!pool || !offs || !level || !blocks || !tgt || (n > 0 && (!off_old || !off_new || !flat || !level_old || !level_new)))
        return GKV_E_NULL;
    gkv::Pool& p = *static_cast<gkv::Pool*>(pool);
    int64_t k = 0, want[gkv::kRungs] = {0};
    for (int64_t row = 0; row < (int64_t)B * Hkv; ++row) {
        const int64_t used = std::min<int64_t>(blocks[row / Hkv], std::min(nb, cap));
        for (int64_t b = 0; b < used; ++b) {
            const int64_t at = row * cap + b;
            int idx;
            if (!gkv::demoted(tgt[row * nb + b], level[at], offs[at], idx)) continue;
            if (k == n) return GKV_E_ARG;
            off_old[k] = offs[at]; flat[k] = at; level_old[k] = level[at]; level_new[k] = gkv::ladder_level(idx);
            ++want[idx]; ++k;
        }
    }
    if (k != n) return GKV_E_ARG;
    if (n == 0) return GKV_OK;
    if (const int rc = gkv::check_alloc(p, want)) return rc;
    int64_t* got = static_cast<int64_t*>(malloc((size_t)n * sizeof(int64_t)));
    if (!got) return GKV_E_MEMORY;
    int64_t start[gkv::kRungs + 1] = {0};
    for (int r = 0; r < gkv::kRungs; ++r) {
        gkv::do_alloc(p, r, want[r], got + start[r]);
        start[r + 1] = start[r] + want[r];
    }
    for (int64_t i = 0; i < n; ++i) off_new[i] = got[start[gkv::ladder_index(level_new[i])]++];
    free(got);
    return GKV_OK;
}

int gkv_table_apply_demotion(void* pool, int64_t* offs, int32_t* level, int64_t n, const int64_t* off_old, const int64_t* off_new,
                             const int64_t* flat, const int32_t* level_old, const int32_t* level_new) {
    if (!pool || !offs || !level || (n > 0 && (!off_old || !off_new || !flat || !level_old || !level_new))) return GKV_E_NULL;
    if (const int rc = gkv::free_by_rung(*static_cast<gkv::Pool*>(pool), off_old, level_old, n)) return rc;
    for (int64_t i = 0; i < n; ++i) { offs[flat[i]] = off_new[i]; level[flat[i]] = level_new[i]; }
    return GKV_OK;
}

}  // extern "C"
