// Tensor-core split decode kernel for the packed bit-ladder cache (sm_100a).
//
// Why tensor cores at all: at HBM speed the 16k-token mix delivers ~7.8e12 codes/s per GPU.
// With a GQA group of 4-8 query heads every code needs 4-8 FMAs plus its unpack, which is
// above the FP32 issue rate of the chip (the CUDA-core kernel in decode_generic.cuh measures
// ~3 % of HBM bandwidth).  The group's QK^T and PV products are therefore issued as
// m16n8k16 MMAs straight from registers; the bytes never make a second trip through shared
// memory, which is why this is mma.sync and not tcgen05 (whose operands must be staged in
// shared memory in canonical layout at 2 B per code).
//
// Structure (one persistent CTA per SM: 12 consumer warps + 2 producer warps + a query warp + a
// scheduler warp):
//   * a small kernel first sorts every cache row's blocks by rung.  A work item is a run of
//     consecutive entries of ONE rung of one row's sorted list (at most kMaxItemBlocks), so an
//     item never mixes rungs: its code path, its query operands and the layout of its
//     accumulators are fixed when it starts.  Items are numbered slot-major (slot * rows + row)
//     and handed out by an atomic counter, so the grid walks the ladder roughly together.  The
//     scheduler warp draws them a few items ahead and parks each item's block table in shared memory;
//   * the blocks of an item alternate between two STREAMS.  Each stream has its own producer
//     warp, its own byte ring in shared memory and three pairs of consumer warps.  The producer
//     starts one bulk copy for a block's bytes and one for its four scale planes, both reporting
//     to the slot's mbarrier (planes that no single copy can collect: 16-byte cp.async);
//   * the query warp turns the next item's query rows into MMA A-fragment planes for the
//     item's rung (double buffered), so the consumers never stop at an item boundary;
//   * a pair of consumer warps takes every third block of its stream and each of its warps
//     one half of the block's tokens (narrow blocks of long items: a warp takes every sixth block),
//     with a private online softmax.  Nothing is merged inside the CTA: the combine kernel merges
//     the per-warp records;
//   * items of centroid blocks (512 bytes each) bypass the rings: the consumer warps read
//     them straight from global memory, sixteen at a time as the MMA fragments of both products.
//
// Arithmetic.  Integer codes are fed to the MMA as fp16 values from the LINEAR range of the
// format: bit patterns 0..2047 (subnormals and the first binade) are worth pattern * 2^-24, so a
// code masked out of the packed word already is the number "code * 2^k * 2^-24" and unpacking
// needs no int->float conversion.  The tensor core aligns the products of a dot product by their
// nominal exponents, so a code sitting in the low mantissa bits wastes that many bits of the
// accumulation window (measured: 2-bit codes at bit 0 lose ~10 bits); codes are therefore
// placed as high in the linear range as a single shift allows and the power of two is folded
// into the other operand or into the epilogue.  De-quantisation is hoisted out of the contraction:
//   q . (c*step + lo) = (q*step) . c + q . lo        (per token group, per channel)
//   p . (c*step + lo) = (p*step) . c + p . lo        (per token, per channel group)
// The small operands q*step and p*step are split into fp16 hi + lo halves (~22 significant
// bits); the lo terms ride along as one more MMA tile on each side.  Accumulation is fp32.
//
// Orientation.  PV is computed TRANSPOSED, O^T[channel][head] (A = value codes, fetched with
// ldmatrix.trans so that a register already holds one channel set of two neighbouring tokens; B =
// p*vstep): 32 accumulator registers per thread instead of 64, which is what lets 12 consumer warps
// share an SM.  With five to eight query heads per cache row QK^T is S[head][token] (A = q*step, hi
// halves in rows 0-7 and lo halves in rows 8-15; B = key codes), which leaves every thread with the
// weights of its head for the token pairs 2t, 2t+1 — exactly a B fragment; PV's hi and lo products
// are two MMAs into the same accumulators.  With at most four heads the eight columns of an MMA hold
// (hi, lo) of every head: QK^T is S[token][head part] (A = key codes), half as many MMAs, a movmatrix
// per eight tokens turns the weights into PV's columns, and one MMA does both halves there too.
//
// What an MMA costs besides its own pipe: on this chip it shares a port with the FP32, HFMA2 and
// integer-multiply pipes.  Per scheduler an m16n8k16 takes 8 cycles, an FP32 instruction 1, HFMA2 and
// IMAD 2, and these ADD UP (one MMA and eight FADDs: 15.5 cycles), while LOP3, PRMT and shifts take
// 2 cycles on a port of their own.  Hence rotations instead of left shifts (rotl), the softmax's
// scales folded into one multiply-add, and fewer MMAs where the shape allows it.
#pragma once

#include <cuda.h>          // CUtensorMap (the type only; the encoder is looked up at run time)

#include "gkv_common.cuh"

namespace gkv {
namespace mma {

// Tensor maps of the cache bytes, one per rung whose blocks are fetched with a TILED bulk copy: the
// cache is described as a byte matrix of `w`-byte rows (w = bytes of a token row, at most 128),
// a block is a box of consecutive rows, and the copy engine writes the box into shared memory with
// the 16-byte chunks of every row XOR-permuted by the row number (the hardware swizzle).  Eight
// consecutive token rows then sit in eight different bank groups, which is what makes the
// ldmatrix.trans fetches of the value codes (eight rows per matrix) conflict-free: measured on the
// plain row-major layout, those fetches alone cost 4 to 8 shared-memory wavefronts per matrix.
//
// A tile row's number is a signed 32-bit coordinate, which rows of 32 bytes exceed from 64 GiB on and rows of 64 bytes from
// 128 GiB on; a copy from beyond it ends in an illegal instruction.  Caches that long are described by lines of 128 bytes,
// each of one, two or four rows: the same bytes in the same order, up to 256 GiB.
constexpr int kLineBytes = 128;     // blocks start on it wherever their sizes are packed without gaps; others are copied by hand
struct alignas(64) TensorMaps {
    CUtensorMap m[3];   // 0: raw bf16 rows, 1: 8-bit codes, 2: 4-bit codes
    CUtensorMap planes; // row form: the four scale planes as (plane, block, bytes), when they lie at equal distances
    int usable;         // 0: no tiled copies (base pointer not 16-byte aligned, or no encoder): blocks are copied by hand
    int planes_tiled;   // 1: `planes` is valid, a block's four planes are one copy
    int lines;          // `m` is (bytes, rows, 1), or 1: (bytes, rows of a line, lines of kLineBytes), for more tile rows than a coordinate counts
    int pad[13];
};

constexpr int kConsumerWarps = 12;       // three warpgroups
constexpr int kStreams = 2;              // byte rings / producer warps per CTA
constexpr int kPairsPerStream = kConsumerWarps / 2 / kStreams;
constexpr int kCtasPerSM = 1;
constexpr int kConsumers = kConsumerWarps * 32;
constexpr int kThreads = kConsumers + 128;          // + helper warpgroup: producers 0/1, query warp, scheduler warp
// Register re-allocation between warpgroups (setmaxnreg): launched with 128 registers per thread
// (512 threads), the helper warpgroup drops to kHelperRegs and the consumers rise to kConsumerRegs:
// 384 * 144 + 128 * 80 = 65536.  (152 and 56 leave the producers short: spills in their loops, 8-bit blocks 218 against 209 us.)
constexpr int kHelperRegs = 80, kConsumerRegs = 144;
#ifndef GKV_K_FETCH
#define GKV_K_FETCH 16    // widest shared-memory load used for a lane's codes of a K row (4, 8 or 16 bytes)
#endif
#ifndef GKV_RING_KB
#define GKV_RING_KB 98    // byte ring per stream
#endif
#ifndef GKV_NSLOT
#define GKV_NSLOT 16
#endif
constexpr int kNSlot = GKV_NSLOT;        // descriptor slots (blocks in flight) per stream
constexpr uint32_t kUnit = 1024;         // ring space is given out in units (the swizzle wants blocks on 1024 bytes)
constexpr uint32_t kRingUnits = GKV_RING_KB;
constexpr uint32_t kRingBytes = kRingUnits * kUnit;
constexpr int kMaxItemBlocks = 128;      // blocks per work item (the item's block table in shared memory)
// Blocks of a centroid item: sixteen are one warp's tile, so items are at least that and twice as long as the others.
__host__ __device__ constexpr int centroid_chunk(int chunk) { return chunk < 8 ? 16 : 2 * chunk < kMaxItemBlocks ? 2 * chunk : kMaxItemBlocks; }
constexpr int kMinItemBlocks = kConsumerWarps / 2;   // one block per pair
constexpr int kItemSlots = 4;            // item descriptors in flight: finishing, current, announced, spare
#ifndef GKV_WAIT_LIMIT_NS
#define GKV_WAIT_LIMIT_NS 1000000000ull
#endif
constexpr unsigned long long kWaitLimitNs = GKV_WAIT_LIMIT_NS;  // every wait gives up after ~1 s, flags the error, returns
constexpr int kPlanTabInts = 8;          // per metadata row: start of each rung class in the sorted list (6), nb, padding

struct Desc {           // one block in a ring
    uint32_t off;       // byte offset of the block in the ring
    int32_t nvalid;
    int32_t pad;
    int32_t orig;       // the block's index in its cache row (for the per-block softmax mass)
};

struct ItemDesc {       // one work item; published one item ahead of its blocks (ring of kItemSlots)
    int32_t item;       // slot * rows + row
    int32_t row;
    int32_t level;      // rung of every block of the item (16, 8, 4, 2, 1)
    int32_t b_lo;       // first entry of the item in the row's sorted list
    int32_t nblk;
    int32_t first;      // stream of the item's first block (blocks alternate from there)
    int32_t end_seq0;   // per stream: the item's blocks are the stream positions below this
    int32_t end_seq1;
    int32_t exit;
    int32_t pad[3];
};

struct Params {
    const float* q;
    const uint8_t* data;
    const __half* klo;
    const __half* kstep;
    const __half* vlo;
    const __half* vstep;
    const uint4* plan;       // (metadata rows, nb) block entries of every row sorted by rung, from plan_kernel
    const int32_t* plan_tab; // (metadata rows, kPlanTabInts) start of each rung class in that list
    float* part;             // (rows, items per row, consumer warps, rep, D): o of every record
    float2* part_ml;         // (rows, items per row, consumer warps, rep): its (m, l)
    float2* mass_part;       // optional (rows, nb, 64 / G units, rep): (reference, sum of weights against it) per unit and head,
                             // natural-log domain; the by-product from which the per-block softmax mass is made
    int* counter;            // work-item counter (zeroed before launch; not read when items are dealt)
    int* status;             // error word (zeroed before launch, or by this kernel: clear_status)
    int B, Hq, Hkv, nb, rep;
    int chunk;               // blocks per item (the last item of a rung's run may be shorter)
    int items_per_row, items;
    int per_row_meta;
    int dealt;               // 1: CTA i takes the items i, i + grid, ...; 0: items are drawn from the counter
    int clear_status;        // 1: this kernel is the first of its call and clears the status word itself
    int rows;
    int paged;               // 1: `data` is a block pool, the lists hold pool offsets, and the four scale planes of a quantised
                             // block sit right behind its bytes ([klo][kstep][vlo][vstep]); klo..vstep above are unused
    int64_t stride_bh;
};

// ---- PTX wrappers --------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, int count) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: false if the phase did not complete within kWaitLimitNs of wall time.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t a = smem_u32(bar);
    unsigned long long t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        uint32_t ok;
        // the hint lets the hardware keep the thread suspended for up to ~2 us before it reports "not yet"
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok) : "r"(a), "r"(parity), "r"(2000u) : "memory");
        if (ok) return true;
#ifndef GKV_NO_BACKOFF
        if (spin > 2) __nanosleep(spin < 64 ? 32 : 256);      // back off: spinning warps steal issue slots
#endif
        if ((spin & 63u) == 63u) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > kWaitLimitNs) return false;
        }
    }
}
// Shared-memory loads by 32-bit shared address (keeps the address arithmetic in 32 bits).
__device__ __forceinline__ uint32_t lds_u8(uint32_t a) { uint32_t v; asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) { uint32_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 lds_v2(uint32_t a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ uint4 lds_v4(uint32_t a) { uint4 v; asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
// Four 8x8 matrices of 16-bit units, transposed: lane L passes the address of row (L & 7) of matrix
// (L >> 3); thread (r = lane >> 2, t = lane & 3) receives, from each matrix, unit r of rows 2t (low
// half) and 2t+1 (high half).
__device__ __forceinline__ void ldsm_x4_trans(uint32_t a, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(a));
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Orders ordinary accesses to shared memory (among them cp.async) before bulk copies that follow, in this thread or
// after a synchronisation with another: barriers alone order accesses of one proxy only.
__device__ __forceinline__ void fence_before_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Arrives on the barrier (without adding to its expected count) when all earlier cp.async of this thread have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// Layout of a rung's block in the ring.  Rungs fetched by a tiled copy are SWIZZLED: byte `off` of the
// block (whose ring address is 1024-byte aligned) lives at off ^ (((off >> 7) & (W/16 - 1)) << 4), W = bytes
// of a tile row (32, 64 or 128) — the 16-byte chunks of a row are permuted by the row's position in
// its group of 128 / W... rows.  W = 0: plain row-major (2-bit codes, and 4-bit codes with 16-channel groups).
template <int D, int G, int BITS>
struct Lay {
    static constexpr int RB = D * BITS / 8;                               // bytes of a token row
    static constexpr bool TILED = BITS == 16 || BITS == 8 || (BITS == 4 && G >= 32);
    static constexpr int W = !TILED ? 0 : RB < 128 ? RB : 128;
    static constexpr uint32_t XMASK = W == 128 ? 7u : W == 64 ? 3u : W == 32 ? 1u : 0u;
    static_assert(!TILED || W >= 32, "tile rows of at least 32 bytes");
};
template <int W>
__device__ __forceinline__ uint32_t swz(uint32_t off) {
    constexpr uint32_t M = W == 128 ? 7u : W == 64 ? 3u : W == 32 ? 1u : 0u;
    return off ^ (((off >> 7) & M) << 4);
}
// XOR term (already shifted to bits 4-6) of a row whose number is r modulo 8, for bytes b of the row
// that do not cross a 128-byte boundary relative to b0.
template <int D, int G, int BITS>
__device__ __forceinline__ uint32_t swz_term(int r, int b0) {
    using L = Lay<D, G, BITS>;
    return ((((uint32_t)r * L::RB + (uint32_t)b0) >> 7) & L::XMASK) << 4;
}

__device__ __forceinline__ void tma_tile3_g2s(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D = A * B (accumulator input zero: the compiler can use the zero register instead of clearing four registers)
__device__ __forceinline__ void mma_f16_z(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_bf16_z(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// w << n for words whose low n bits are masked out afterwards: a rotation goes to the integer pipe, while the compiler likes to
// make multiplications of shifts, on the pipe that the MMAs keep busy.
__device__ __forceinline__ uint32_t rotl(uint32_t w, int n) { return n ? __funnelshift_l(w, w, n) : w; }

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// (x*y) as fp16 hi + lo, x given as fp16 hi/lo halves, y exact fp16: hi = rn(xh*y),
// lo = rn(xl*y + (xh*y - hi)); the inner difference is exact in an fp16 FMA.
__device__ __forceinline__ void mul_split(uint32_t xh, uint32_t xl, uint32_t y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __hmul2(u32_as_h2(xh), u32_as_h2(y));
    const __half2 e = __hfma2(u32_as_h2(xh), u32_as_h2(y), __hneg2(h));
    hi = h2_as_u32(h);
    lo = h2_as_u32(__hfma2(u32_as_h2(xl), u32_as_h2(y), e));
}

// Two fp32 values -> packed fp16 hi pair and residual lo pair (element 0 in the low half).
__device__ __forceinline__ void split_f16x2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 hf = __half22float2(h);
    hi = h2_as_u32(h);
    lo = h2_as_u32(__floats2half2_rn(x0 - hf.x, x1 - hf.y));
}
__device__ __forceinline__ void split_bf16x2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
    const float2 hf = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x0 - hf.x, x1 - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// ---- channel arrangement of the QK contraction -----------------------------------------------
// Thread t of a quad owns DT = D/4 consecutive channels of a token row.  MMA k-step s, slot e
// (e = 0,1 -> first B register, e = 2,3 -> second) maps to channel DT*t + arr_chan(bits, s, e);
// the maps follow the cheapest shift-and-mask unpack of each code width (one 32-bit AND yields
// the two codes that sit 16 bits apart).  arr_scale is the exact power of two folded into the
// prepared query so that every slot of a rung carries the same weight:
//   4-bit: even nibbles land on bits 3-6 (8c), odd nibbles on bits 7-10 (128c)  -> x16 / x1
//   2-bit: even fields land on bits 8-9 (256c), odd fields on bits 6-7 (64c)    -> x1 / x4
__host__ __device__ constexpr int arr_chan(int bits, int s, int e) {
    return bits == 4   ? 8 * (s >> 1) + 2 * (s & 1) + (e >> 1) + 4 * (e & 1)
           : bits == 2 ? 16 * (s >> 2) + 2 * (s & 3) + (e >> 1) + 8 * (e & 1)
                       : 4 * s + e;   // 8-bit codes and raw bf16
}
__host__ __device__ constexpr float arr_scale(int bits, int e) {
    return bits == 4 ? ((e >> 1) ? 1.f : 16.f) : bits == 2 ? ((e >> 1) ? 4.f : 1.f) : 1.f;
}
// 2^24 / (weight of one code in the linear range) for the K contraction of each rung
__host__ __device__ constexpr float k_unscale(int bits) { return bits == 4 ? 131072.f : bits == 2 ? 65536.f : 16777216.f; }

// Head whose scores a thread with row index r (= lane >> 2) holds.  With at most four heads per
// cache row, rows 2h and 2h+1 both carry head h, so that the two threads can feed the hi and the
// lo column of that head in the transposed PV product.
template <bool DUP>
__device__ __forceinline__ int head_of_row(int r) { return DUP ? (r >> 1) : r; }

template <int D, int G>
struct Cfg {
    static constexpr int DT = D / 4;          // channels per thread in QK
    static constexpr int KS = D / 16;         // QK k-steps
    static constexpr int CH = KS / 2;         // 16-byte chunks of prepared q per thread (2 k-steps each)
    static constexpr int TG = kP / G;         // token groups (K scales)
    static constexpr int GV = D / G;          // channel groups (V scales)
    static constexpr int MT = D / 16;         // output m-tiles (16 channels each) of the transposed PV product
    static constexpr int KSCALE = TG * D * 2; // bytes of klo (or kstep) of one block
    static constexpr int VSCALE = kP * GV * 2;
    // prepared-q planes, in halves: [plane][chunk][lane][8], in the channel arrangement of the item's rung (query_planes)
    static constexpr int QPLANE = CH * 32 * 8;
    static constexpr int QPREP_BYTES = 3 * QPLANE * 2;
    static constexpr int SQ_BYTES = 8 * D * 4;
    static constexpr size_t SMEM = 1024 + kStreams * (size_t)kRingBytes + 2 * (QPREP_BYTES + SQ_BYTES + 64) +
                                   kStreams * kNSlot * (sizeof(Desc) + 16) + kItemSlots * sizeof(ItemDesc) +
                                   (2 * kItemSlots + 2) * 8 + kItemSlots * kMaxItemBlocks * 16 + 128;
    static_assert(D % 32 == 0 && (G == 16 || G == 32 || G == 64) && D % G == 0, "unsupported shape");
};

template <int D, int G>
struct Smem {
    using C = Cfg<D, G>;
    uint8_t* ring;         // [kStreams][kRingBytes]
    __half* qprep;         // [2] prepared-query planes (item parity)
    float* sq;             // [2][8][D] raw query (fp32, softmax scale included)
    float* sf;             // [2][16]: per-head factor 2^-eq * log2(e), then 2^eq
    Desc* desc;            // [kStreams][kNSlot]
    uint64_t* full;        // [kStreams][kNSlot]
    uint64_t* empty;       // [kStreams][kNSlot]
    ItemDesc* item;        // [kItemSlots]
    uint64_t* item_full;   // [kItemSlots] scheduler warp -> producers, query warp and consumers
    uint64_t* item_empty;  // [kItemSlots] one arrival per consumer warp and per producer that is done with the item
    uint64_t* qready;      // [2] query warp -> consumers
    uint4* item_tab;       // [kItemSlots][kMaxItemBlocks] block entries of the announced items (row base offset added)
    __device__ explicit Smem(uint8_t* raw) {
        // the swizzle of the tiled copies is a function of the shared-memory address: rings start on a 1024-byte boundary
        uint8_t* base = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
        ring = base;
        uint8_t* p = base + kStreams * (size_t)kRingBytes;
        qprep = reinterpret_cast<__half*>(p);               p += 2 * C::QPREP_BYTES;
        sq = reinterpret_cast<float*>(p);                   p += 2 * C::SQ_BYTES;
        sf = reinterpret_cast<float*>(p);                   p += 2 * 16 * 4;
        item_tab = reinterpret_cast<uint4*>(p);             p += kItemSlots * kMaxItemBlocks * 16;
        item = reinterpret_cast<ItemDesc*>(p);              p += kItemSlots * sizeof(ItemDesc);
        desc = reinterpret_cast<Desc*>(p);                  p += kStreams * kNSlot * sizeof(Desc);
        full = reinterpret_cast<uint64_t*>(p);              p += kStreams * kNSlot * 8;
        empty = reinterpret_cast<uint64_t*>(p);             p += kStreams * kNSlot * 8;
        item_full = reinterpret_cast<uint64_t*>(p);         p += kItemSlots * 8;
        item_empty = reinterpret_cast<uint64_t*>(p);        p += kItemSlots * 8;
        qready = reinterpret_cast<uint64_t*>(p);
    }
};

// ---- launches that overlap ---------------------------------------------------------------------------
// The kernels of a call follow one another in a stream, and each may be launched before its predecessor has ended
// (programmatic dependent launch): a small kernel lets its dependents start as soon as all of its own CTAs run, the
// split kernel when its CTAs end (merge CTAs that wait on the SMs that finish first made a call 2 to 4 % slower),
// and every kernel waits (grid_wait: until its predecessor has ended and its writes are visible) before it touches
// anything the predecessor wrote.  What overlaps is launch latency and set-up: one 16k-token sequence 36.4 -> 28.1 us
// per call, six short ones in a pool 39.1 -> 33.6 us.
// The first kernel of a call is launched the ordinary way, so nothing of a call starts before the stream's earlier work
// (the query, the workspace's last readers) is done.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Work counter and status word of a call whose block lists are kept by the caller (plan_kernel does it otherwise).
__global__ void reset_kernel(int* header, int header_ints) {
    grid_release();
    if ((int)threadIdx.x < header_ints) header[threadIdx.x] = 0;
}

// ---- rung-sorted block lists -----------------------------------------------------------------------
// One CTA per metadata row: a stable counting sort of the row's blocks by rung (16, 8, 4, 2,
// centroid, then blocks with nothing to do).  An entry is everything the producer needs to know
// about a block: byte offset in the row (64 bit), level | nvalid << 8 (level 0: skip), block index.
// Every thread owns a contiguous run of blocks, counts its classes, an in-order scan over
// (class, thread) gives it a write cursor per class, and it walks its run once more.  Deterministic:
// no atomics.  The start of every class in the list goes to the row's table.  Also clears the
// workspace header when given one.
constexpr int kPlanMaxThreads = 1024;
__device__ __forceinline__ int rung_class(int lv, int nv) {
    return nv <= 0 ? 5 : lv == 16 ? 0 : lv == 8 ? 1 : lv == 4 ? 2 : lv == 2 ? 3 : lv == 1 ? 4 : 5;
}
__global__ void __launch_bounds__(kPlanMaxThreads) plan_kernel(const int32_t* level, const int32_t* valid, const int64_t* offs,
                                                                uint4* plan, int32_t* plan_tab, int nb, int* header,
                                                                int header_ints) {
    grid_release();
    // the decode kernel's work counter and status word start at zero
    if (blockIdx.x == 0 && header)
        for (int i = threadIdx.x; i < header_ints; i += blockDim.x) header[i] = 0;
    __shared__ int wsum[kPlanMaxThreads / 32][6];   // per-warp class totals, then their exclusive scan
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    const int32_t* lv = level + (size_t)blockIdx.x * nb;
    const int32_t* nv = valid + (size_t)blockIdx.x * nb;
    const int64_t* of = offs + (size_t)blockIdx.x * nb;
    uint4* out = plan + (size_t)blockIdx.x * nb;
    const int per = (nb + (int)blockDim.x - 1) / (int)blockDim.x;
    const int lo = min(nb, tid * per), hi = min(nb, lo + per);
    // rows of at most kPlanMaxThreads blocks have one block per thread: it is read once and kept
    int lv0 = 0, nv0 = 0, cls0 = 5;
    unsigned long long of0 = 0;
    int cnt[6] = {0, 0, 0, 0, 0, 0};
    if (per == 1) {
        if (lo < hi) { lv0 = lv[lo]; nv0 = nv[lo]; of0 = (unsigned long long)of[lo]; }
        cls0 = rung_class(lv0, nv0);
#pragma unroll
        for (int k = 0; k < 6; ++k) cnt[k] = (lo < hi && cls0 == k);
    } else {
        for (int b = lo; b < hi; ++b) {
            const int c = rung_class(lv[b], nv[b]);
#pragma unroll
            for (int k = 0; k < 6; ++k) cnt[k] += (c == k);
        }
    }
    int cur[6];                                     // exclusive prefix inside the warp
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        int x = cnt[k];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        cur[k] = x - cnt[k];
        if (lane == 31) wsum[warp][k] = x;
    }
    __syncthreads();
    // every warp scans the (at most 32) warps' totals for itself: no second barrier, no serial walk over them
    int run = 0, first[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int mine = lane < nwarp ? wsum[lane][k] : 0;
        int x = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        first[k] = run;                             // class k occupies [first[k], first[k+1]) of the list
        cur[k] += run + __shfl_sync(0xffffffffu, x - mine, warp);
        run += __shfl_sync(0xffffffffu, x, 31);
    }
    if (tid == 0) {
        int32_t* tab = plan_tab + (size_t)blockIdx.x * kPlanTabInts;
#pragma unroll
        for (int k = 0; k < 6; ++k) tab[k] = first[k];
        tab[6] = nb; tab[7] = 0;
    }
    if (per == 1) {
        if (lo < hi) {
            const int n = min(nv0, kP);
            const uint4 e = make_uint4((uint32_t)of0, (uint32_t)(of0 >> 32), cls0 == 5 ? 0u : ((uint32_t)lv0 | ((uint32_t)n << 8)), (uint32_t)lo);
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (cls0 == k) out[cur[k]] = e;
        }
        return;
    }
    for (int b = lo; b < hi; ++b) {
        const int l = lv[b], n = min(nv[b], kP);
        const int c = rung_class(l, n);
        const unsigned long long o = (unsigned long long)of[b];
        const uint4 e = make_uint4((uint32_t)o, (uint32_t)(o >> 32), c == 5 ? 0u : ((uint32_t)l | ((uint32_t)n << 8)), (uint32_t)b);
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (c == k) out[cur[k]++] = e;
    }
}

// ================================ producers ===================================================
// Item `id` = slot * rows + row.  Slot s of a row is the s-th chunk when each rung's run of the
// row's sorted list is cut into chunks of p.chunk blocks; slots beyond the row's last chunk are
// empty (rows have a fixed number of slots, enough for any mix of rungs).
struct Span { int row, level, b_lo, nblk; };
__device__ __forceinline__ Span span_of(const Params& p, int id) {
    Span sp{0, 0, 0, 0};
    if (id >= p.items) return sp;
    int slot = id / p.rows;
    sp.row = id % p.rows;
    const int32_t* tab = p.plan_tab + (size_t)(p.per_row_meta ? sp.row : 0) * kPlanTabInts;
    // Items are handed out slot by slot over all rows, so at any moment the whole grid works on the same
    // slot index: every row walks its rungs 16, 8, 4, 2, centroid — the costliest items first, the
    // cheapest in the tail.  (Letting odd rows walk 4, 2, 16, 8, centroid, so that some SMs stream wide
    // blocks while others unpack narrow ones, measured 12 % slower on the 16k-token workload.)
    // the row's six class starts in two loads (the table rows are 32 bytes, aligned): one round trip per
    // drawn item instead of one per class walked
    const int4 t0 = *reinterpret_cast<const int4*>(tab);
    const int2 t1 = *reinterpret_cast<const int2*>(tab + 4);
    const int st[6] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int start = st[k], cnt = st[k + 1] - start;
        const int ck = k == 4 ? centroid_chunk(p.chunk) : p.chunk;
        const int n = (cnt + ck - 1) / ck;
        if (slot < n) {
            sp.level = ladder_level(k);
            sp.b_lo = start + slot * ck;
            sp.nblk = min(ck, cnt - slot * ck);
            return sp;
        }
        slot -= n;
    }
    return sp;
}

struct ProducerState {
    uint32_t head = 0;                  // where the next block goes, in kUnit bytes of the ring
    uint32_t vhead = 0, vtail = 0;      // units allocated and released since the start (waste at the wrap included)
    uint32_t vend = 0;                  // lane s < kNSlot: vhead behind the block in slot s
    int seq_alloc = 0, seq_free = 0;
};

// Non-blocking test of a barrier phase.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

// One stream's blocks of one item, in BATCHES.  A producer warp shares its scheduler with three consumer warps and gets an
// instruction in every eight cycles or so: what it costs is the length of its chain, and with ~1300 cycles per block (a loop
// over the released slots, another over the blocks that fit, shuffles per block, a division) it was what bounded blocks of
// eight bits and less.  So nothing here is done block by block except the copies themselves: lane i tests slot i of those in
// flight; an item's blocks are all of one size, so how many fit and where block i goes is arithmetic; lane i then publishes
// block i of the batch, arms its barrier and starts ONE copy for its bytes and one for the scale planes of a quantised rung.
// In the pool form the planes follow the block (2-bit blocks: one copy for both); in the row form they are four tensors, which
// one tiled copy collects when they lie at equal distances (as pack_cache lays them out).  Other planes are fetched by all 32
// lanes with 16-byte asynchronous copies that arrive on the same barrier: about 500 cycles per block, of which the 32 arrivals
// take 200; one bulk copy per plane costs as much, and so did a warp of its own for them (4-bit blocks 180 -> 203 us).
template <int D, int G>
__device__ __forceinline__ bool produce_item(const Params& p, const TensorMaps& tm, Smem<D, G>& sm, ProducerState& ps, int s,
                                             const ItemDesc& it, int islot) {
    using C = Cfg<D, G>;
    const int lane = threadIdx.x & 31;
    if (it.level == 1 || it.nblk == 0) return true;     // centroid items are read straight from global memory
    const int j0 = (s ^ it.first) & 1;                   // this stream's first block of the item
    const int n_mine = (it.nblk - j0 + 1) >> 1;
    const uint32_t tab = smem_u32(sm.item_tab + islot * kMaxItemBlocks + j0);      // this stream's blocks: every second entry
    const int lv = it.level;
    const bool quant = lv != 16;
    const bool by_lanes = !p.paged && !tm.planes_tiled;  // (see the comment above)
    const uint32_t dbytes = 2u * (uint32_t)half_bytes(lv, D);
    constexpr int K = C::KSCALE;                         // == VSCALE: every scale plane has the same bytes per block
    static_assert(C::KSCALE == C::VSCALE && (4 * K) % 512 == 0, "scale planes");
    constexpr int NR = 4 * K / 512;                      // rounds of 32 lanes x 16 bytes that cover the four planes
    const uint32_t need = (dbytes + (quant ? 4u * K : 0u) + kUnit - 1) / kUnit;
    const uint32_t inv = (65536u + need - 1) / need;     // x * inv >> 16 == x / need for x <= kRingUnits
    // tiled copies: log2 of the tile row width of the item's rung (0: plain bulk copy) and its tensor map
    constexpr int W4 = Lay<D, G, 4>::W;
    const int tw = lv == 16 ? Lay<D, G, 16>::W : lv == 8 ? Lay<D, G, 8>::W : lv == 4 ? W4 : 0;
    const int at_shift = tw == 128 || tm.lines ? 7 : tw == 64 ? 6 : 5;
    const unsigned long long at_mask = (1ull << at_shift) - 1;
    const CUtensorMap* tmap = &tm.m[lv == 16 ? 0 : lv == 8 ? 1 : 2];
    uint64_t* full = sm.full + s * kNSlot;
    uint64_t* empty = sm.empty + s * kNSlot;
    Desc* desc = sm.desc + s * kNSlot;
    const uint32_t ring = smem_u32(sm.ring) + (uint32_t)s * kRingBytes;
    for (int j = 0; j < n_mine;) {
        // slots the consumers are done with, oldest first
        {
            const int seq = ps.seq_free + lane;
            const bool done = seq < ps.seq_alloc && mbar_test(&empty[seq % kNSlot], (uint32_t)(seq / kNSlot) & 1u);
            const int n = __ffs(~__ballot_sync(0xffffffffu, done)) - 1;          // at most kNSlot are in flight
            const uint32_t end = __shfl_sync(0xffffffffu, ps.vend, (ps.seq_free + n - 1) & (kNSlot - 1));
            if (n > 0) { ps.vtail = end; ps.seq_free += n; }
        }
        // how many of the next blocks fit: n1 up to the end of the ring, n2 from its start
        const int want = min(n_mine - j, kNSlot - (ps.seq_alloc - ps.seq_free));
        const uint32_t room = kRingUnits - (ps.vhead - ps.vtail);
        const int k1 = (int)(((kRingUnits - ps.head) * inv) >> 16);
        const int n1 = min(min(want, k1), (int)((room * inv) >> 16));
        const uint32_t waste = kRingUnits - ps.head - (uint32_t)k1 * need;
        const int rest = (int)room - (int)(kRingUnits - ps.head);        // free units behind the wrap
        const int n2 = n1 == k1 && rest > 0 ? min(want - n1, (int)(((uint32_t)rest * inv) >> 16)) : 0;
        const int nfit = n1 + n2;
        if (nfit == 0) {                                 // nothing fits: wait for the oldest block to be released
            const int sl = ps.seq_free % kNSlot;
            if (!mbar_wait(&empty[sl], (uint32_t)(ps.seq_free / kNSlot) & 1u)) return false;
            continue;
        }
        const uint32_t head = ps.head;
        auto place = [&](int i) { return (i < n1 ? head + (uint32_t)i * need : (uint32_t)(i - n1) * need) * kUnit; };
        {
            const int i = (lane - ps.seq_alloc) & (kNSlot - 1);          // the block of the batch that takes slot `lane`
            if (i < nfit) ps.vend = ps.vhead + (uint32_t)(i + 1) * need + (i >= n1 ? waste : 0u);
            ps.vhead += (uint32_t)nfit * need + (n2 ? waste : 0u);
            ps.head = n2 ? (uint32_t)n2 * need : head + (uint32_t)n1 * need;
            if (ps.head == kRingUnits) ps.head = 0;
        }
        // What the lanes have seen released, all of them have (the warp barrier); and the copies below may land on bytes that
        // ordinary stores put there (planes and blocks copied by this warp's lanes, cleared tails): every lane fences before
        // the copy it starts: one fence per batch here, not one per block in the warps that release the slots.
        __syncwarp();
        fence_before_bulk();
        bool withhold = false;
        if (lane < nfit) {
            const int my_seq = ps.seq_alloc + lane, my_slot = my_seq % kNSlot;
            const uint32_t my_dst = place(lane);
            const uint4 cur = lds_v4(tab + 32u * (uint32_t)(j + lane));
#ifdef GKV_TEST_WITHHOLD_BLOCK
            // test build only: the second block of stream 0 never arrives, so the waits on it run out
            withhold = s == 0 && my_seq == 1;
#endif
            Desc d;
            d.off = my_dst; d.nvalid = (int)((cur.z >> 8) & 0xffu); d.orig = (int32_t)cur.w; d.pad = 0;
            desc[my_slot] = d;
            const unsigned long long soff = ((unsigned long long)cur.y << 32) | cur.x;      // byte offset in the cache
            const uint8_t* src = p.data + soff;
            if (withhold) {
            } else {
                // where the lanes fetch planes a barrier expects 32 arrivals more: theirs, or all at once for a block without planes
                if (by_lanes && !quant) mbar_arrive_n(&full[my_slot], 32);
                const uint32_t planes = quant && !by_lanes ? 4u * K : 0u;        // planes that a copy of this lane's brings
                const uint32_t behind = p.paged ? planes : 0u;                   // ... from behind the block
                if (planes && !p.paged) {
                    mbar_expect_tx(&full[my_slot], planes);
                    tma_tile3_g2s(ring + my_dst + dbytes, &tm.planes, 0, it.row * p.nb + (int)cur.w, 0, &full[my_slot]);
                }
                if (tw && tm.usable && (soff & at_mask) == 0) {
                    // a box of tile rows, written swizzled (row = byte offset / row width)
                    mbar_arrive_tx(&full[my_slot], dbytes + behind);
                    const int at = (int)(soff >> at_shift);
                    tma_tile3_g2s(ring + my_dst, tmap, 0, tm.lines ? 0 : at, tm.lines ? at : 0, &full[my_slot]);
                    if (behind) bulk_g2s(ring + my_dst + dbytes, src + dbytes, behind, &full[my_slot]);
                } else if (!tw && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
                    mbar_arrive_tx(&full[my_slot], dbytes + behind);
                    bulk_g2s(ring + my_dst, src, dbytes + behind, &full[my_slot]);
                } else {
                    // block start not aligned for a bulk copy (a cache row at an odd address): this lane
                    // copies the bytes by hand, into the layout the rung's consumers expect
                    uint8_t* d0 = sm.ring + (size_t)s * kRingBytes + my_dst;
                    if (tw == 128) for (uint32_t i = 0; i < dbytes; ++i) d0[swz<128>(i)] = src[i];
                    else if (tw == 64) for (uint32_t i = 0; i < dbytes; ++i) d0[swz<64>(i)] = src[i];
                    else if (tw == 32) for (uint32_t i = 0; i < dbytes; ++i) d0[swz<32>(i)] = src[i];
                    else for (uint32_t i = 0; i < dbytes; ++i) d0[i] = src[i];
                    for (uint32_t i = 0; i < behind; ++i) d0[dbytes + i] = src[dbytes + i];
                    __threadfence_block();
                    mbar_arrive(&full[my_slot]);
                }
            }
        }
        if (quant && by_lanes) {
            const unsigned held = __ballot_sync(0xffffffffu, withhold);
#pragma unroll 2
            for (int i = 0; i < nfit; ++i) {
                if ((held >> i) & 1u) continue;
                const size_t so = ((size_t)it.row * p.nb + lds_u32(tab + 32u * (uint32_t)(j + i) + 12u)) * K;
                const uint32_t sdst = ring + place(i) + dbytes + (uint32_t)lane * 16u;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const int o = r * 512 + lane * 16, which = o / K;            // 0 klo, 1 kstep, 2 vlo, 3 vstep
                    const uint8_t* base = reinterpret_cast<const uint8_t*>(which == 0 ? p.klo : which == 1 ? p.kstep
                                                                           : which == 2 ? p.vlo : p.vstep);
                    cp_async16(sdst + (uint32_t)(r * 512), base + so + (o - which * K));
                }
                cp_async_arrive(&full[(ps.seq_alloc + i) % kNSlot]);     // one arrival per lane once its copies have landed
            }
        }
        __syncwarp();
        ps.seq_alloc += nfit;
        j += nfit;
    }
    return true;
}

// The scheduler warp draws the work items (an atomic counter), looks up what each one is, fetches
// its block entries into the item's table in shared memory and announces it — up to kItemSlots - 1
// items ahead of the consumers, so none of this global-memory latency is ever waited for by the
// producers or the consumers.  Items without blocks are not announced, and nothing is written to their records: the merge
// works out how many of a row's records exist and reads no others.
template <int D, int G>
__device__ void scheduler_loop(const Params& p, Smem<D, G>& sm, int* abort_flag) {
    const int lane = threadIdx.x & 31;
    int tot0 = 0, tot1 = 0, nfirst = 0, drawn = 0;
    bool ok = true;
    grid_wait();            // block lists, work counter and status word: this warp alone reads the first two, and everything
                            // the other warps do follows from what it announces
    if (p.clear_status && blockIdx.x == 0 && lane == 0) *p.status = 0;      // whoever gives up sets it after milliseconds of waiting
    for (int j = 0; ok; ++j) {
        ItemDesc it;
        for (;;) {                                          // draw the next item that has blocks
            int id = 0;
            if (p.dealt) id = (int)blockIdx.x + (int)gridDim.x * drawn++;
            else {
                if (lane == 0) id = atomicAdd(p.counter, 1);
                id = __shfl_sync(0xffffffffu, id, 0);
            }
            const Span sp = span_of(p, id);                 // same loads in every lane (broadcast)
            it.item = id; it.row = sp.row; it.level = sp.level; it.b_lo = sp.b_lo; it.nblk = sp.nblk;
            it.exit = id >= p.items ? 1 : 0;
            it.pad[0] = it.pad[1] = it.pad[2] = 0;
            if (it.exit || sp.nblk > 0) break;
            // an empty slot of the row: nothing to do and nothing to write — the used slots of a row are a
            // prefix of its slots, and the merge kernel works out from the row's class counts how many
            // there are, so it never reads the records of an empty slot
        }
        it.first = nfirst & 1;
        if (!it.exit && it.level != 1) {
            const int n0 = (it.nblk + 1) >> 1, n1 = it.nblk >> 1;       // the first stream gets the odd block
            if (it.first) { tot1 += n0; tot0 += n1; } else { tot0 += n0; tot1 += n1; }
            ++nfirst;
        }
        it.end_seq0 = tot0;
        it.end_seq1 = tot1;
        // the item's block entries, four per lane, with the row's base offset added
        constexpr int kPerLane = kMaxItemBlocks / 32;
        uint4 e[kPerLane];
#pragma unroll
        for (int h = 0; h < kPerLane; ++h) {
            e[h] = make_uint4(0, 0, 0, 0);
            const int i = lane + 32 * h;
            if (!it.exit && i < it.nblk) {
                e[h] = p.plan[(size_t)(p.per_row_meta ? it.row : 0) * p.nb + it.b_lo + i];
                const unsigned long long src = (unsigned long long)it.row * (unsigned long long)p.stride_bh +
                                               (((unsigned long long)e[h].y << 32) | e[h].x);
                e[h].x = (uint32_t)src; e[h].y = (uint32_t)(src >> 32);
            }
        }
        // the descriptor slot is free once everybody has finished item j - kItemSlots
        const int sl = j % kItemSlots;
        if (j >= kItemSlots) ok = mbar_wait(&sm.item_empty[sl], (uint32_t)(j / kItemSlots - 1) & 1u);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < kPerLane; ++h) sm.item_tab[sl * kMaxItemBlocks + lane + 32 * h] = e[h];
        if (lane == 0) sm.item[sl] = it;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.item_full[sl]);
        if (it.exit) return;
        if (*reinterpret_cast<volatile int*>(abort_flag)) return;
    }
    if (!ok && lane == 0) {
        atomicExch(p.status, 1);
        atomicExch(abort_flag, 1);
    }
}

// Producer of stream s: for every announced item, streams the item's blocks of its stream into its ring.
template <int D, int G>
__device__ void producer_loop(const Params& p, const TensorMaps& tm, Smem<D, G>& sm, int s, int* abort_flag) {
    const int lane = threadIdx.x & 31;
    ProducerState ps;
    bool ok = true;
    for (int j = 0; ok; ++j) {
        const int sl = j % kItemSlots;
        if (!mbar_wait(&sm.item_full[sl], (uint32_t)(j / kItemSlots) & 1u)) { ok = false; break; }
        const ItemDesc it = sm.item[sl];
        if (it.exit) return;
        ok = produce_item<D, G>(p, tm, sm, ps, s, it, sl);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.item_empty[sl]);      // this warp no longer needs the item's descriptor and table
        if (*reinterpret_cast<volatile int*>(abort_flag)) return;
    }
    if (!ok && lane == 0) {
        atomicExch(p.status, 9 + s);
        atomicExch(abort_flag, 1);
    }
}

// ================================ query warp ==================================================
// For every announced item: the row's query heads, a per-head
// power-of-two scale, and the MMA A-fragment planes (hi, lo) in the channel arrangement of the
// item's rung, into the buffer of the item's parity.  Runs one item ahead of the consumers.
//
// What bounds it is its own latency, which every short item and the start of every call wait for, so: the row arrives
// by one round of 16-byte loads (requested before the buffer is known to be free), the heads' maxima are reduced
// side by side in registers, and the planes are written by code for the item's rung, two 16-byte loads per chunk.
// Measured: the split kernel of a six-row batch of short sequences 14.5 -> 10.9 us.
template <int D, int G, bool DUP, int BITS>
__device__ __forceinline__ void query_planes(const float* sq, const float* sf, __half* qp) {
    using C = Cfg<D, G>;
    // This lane writes its own fragment lane of every chunk: 8 halves (two k-steps x four slots) per plane and chunk,
    // as one 16-byte store.
    const int lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
    const int head = head_of_row<DUP>(r);
    const float sc = sf[8 + head];
    const float* qr = sq + head * D + C::DT * t;
#pragma unroll
    for (int i = 0; i < C::CH; ++i) {
        // the chunk's eight channels: two runs of four
        constexpr int kGap = BITS == 2 ? 8 : 4;
        const int c0 = BITS == 2 ? 16 * (i >> 1) + 4 * (i & 1) : 8 * i;
        const float4 lo4 = *reinterpret_cast<const float4*>(qr + c0), hi4 = *reinterpret_cast<const float4*>(qr + c0 + kGap);
        const float x[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int jp = 0; jp < 4; ++jp) {            // halves 2jp, 2jp+1: k-step 2i + (jp >> 1), slots 2(jp & 1) + {0, 1}
            const int ks = 2 * i + (jp >> 1), e0 = 2 * (jp & 1);
            const int a0 = arr_chan(BITS, ks, e0) - c0, a1 = arr_chan(BITS, ks, e0 + 1) - c0;
            const float x0 = x[a0 >= kGap ? a0 - kGap + 4 : a0] * sc * arr_scale(BITS, e0);
            const float x1 = x[a1 >= kGap ? a1 - kGap + 4 : a1] * sc * arr_scale(BITS, e0 + 1);
            if (BITS != 16) split_f16x2(x0, x1, hi[jp], lo[jp]);
            else split_bf16x2(x0, x1, hi[jp], lo[jp]);
        }
        uint4* dst = reinterpret_cast<uint4*>(qp + ((size_t)i * 32 + lane) * 8);
        if (!DUP) {
            dst[0] = make_uint4(hi[0], lo[0], hi[1], lo[1]);                 // A registers a0..a3 of k-step 2i
            dst[C::QPLANE / 8] = make_uint4(hi[2], lo[2], hi[3], lo[3]);     // ... and of k-step 2i+1
        } else if (BITS == 16) {                                             // B registers of k-steps 2i and 2i+1
            dst[0] = (r & 1) ? make_uint4(lo[0], lo[1], lo[2], lo[3]) : make_uint4(hi[0], hi[1], hi[2], hi[3]);
        } else {                                                             // operands of mul_part for the same registers
            constexpr uint32_t kNeg = 0x80008000u;
            const uint32_t on = (r & 1) ? 0xffffffffu : 0u;
            dst[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            dst[C::QPLANE / 8] = make_uint4((hi[0] ^ kNeg) & on, (hi[1] ^ kNeg) & on, (hi[2] ^ kNeg) & on, (hi[3] ^ kNeg) & on);
            dst[2 * C::QPLANE / 8] = make_uint4(lo[0] & on, lo[1] & on, lo[2] & on, lo[3] & on);
        }
    }
}

template <int D, int G, bool DUP>
__device__ void query_loop(const Params& p, Smem<D, G>& sm, int* abort_flag) {
    using C = Cfg<D, G>;
    constexpr int LPR = D / 4;                  // lanes that cover a head's row with four channels each (32 or 16)
    constexpr int NV = 8 * LPR / 32;            // 16-byte loads per lane for eight heads
    const int lane = threadIdx.x & 31;
    int code = 0;
    for (int j = 0;; ++j) {
        const int s = j % kItemSlots, ib = j & 1;
        if (!mbar_wait(&sm.item_full[s], (uint32_t)(j / kItemSlots) & 1u)) { code = 7; break; }
        const ItemDesc it = sm.item[s];
        if (it.exit) return;
        const int b = it.row / p.Hkv, hk = it.row % p.Hkv;
        const float* q = p.q + ((size_t)b * p.Hq + (size_t)hk * p.rep) * D;
        float4 v[NV];
        const bool wide = (reinterpret_cast<uintptr_t>(q) & 15) == 0;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int e = (i * 32 + lane) * 4;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (e / D < p.rep) {
                if (wide) v[i] = __ldg(reinterpret_cast<const float4*>(q + e));
                else v[i] = make_float4(q[e], q[e + 1], q[e + 2], q[e + 3]);
            }
        }
        // the query buffer was last used by item j-2: wait until every consumer warp has left it
        if (j >= 2 && !mbar_wait(&sm.item_empty[(j - 2) % kItemSlots], (uint32_t)((j - 2) / kItemSlots) & 1u)) { code = 8; break; }
        float* sq = sm.sq + ib * 8 * D;
        float* sf = sm.sf + ib * 16;
        __half* qp = sm.qprep + (size_t)ib * (C::QPREP_BYTES / 2);
#pragma unroll
        for (int i = 0; i < NV; ++i) *reinterpret_cast<float4*>(sq + (i * 32 + lane) * 4) = v[i];
        {
            // per-head power-of-two scale bringing max|q| into [8, 16); lane h ends up with head h's maximum
            float top = 0.f;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                float mx = fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
#pragma unroll
                for (int o = LPR / 2; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                if (LPR == 32) {
                    if (lane == i) top = mx;
                } else {
                    const float other = __shfl_sync(0xffffffffu, mx, (lane & 1) * LPR);      // heads 2i and 2i+1
                    if ((lane >> 1) == i) top = other;
                }
            }
            if (lane < 8) {
                int eq = 0;
                if (top > 0.f && top < INFINITY) eq = 3 - ilogbf(top);
                eq = max(-100, min(100, eq));
                sf[lane] = ldexpf(1.4426950408889634f, -eq);
                sf[8 + lane] = ldexpf(1.0f, eq);
            }
            __syncwarp();
            if (it.level == 1) query_planes<D, G, false, 8>(sq, sf, qp);          // fp16 rows: heads are rows for any number of them
            else if (it.level == 16) query_planes<D, G, DUP, 16>(sq, sf, qp);
            else if (it.level == 8) query_planes<D, G, DUP, 8>(sq, sf, qp);
            else if (it.level == 4) query_planes<D, G, DUP, 4>(sq, sf, qp);
            else query_planes<D, G, DUP, 2>(sq, sf, qp);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.qready[ib]);
    }
    if (lane == 0) {
        atomicExch(p.status, code);
        atomicExch(abort_flag, 1);
    }
}

// ================================ consumers ===================================================
// The blocks are processed in UNITS of G tokens (one token group of the K scales): scores of
// the unit, online-softmax update, value product of the unit.  All shared-memory operands are
// addressed by 32-bit shared addresses built from one per-thread base plus compile-time offsets.
template <int D, int G>
struct Unit {
    static constexpr int U = G;          // tokens
    static constexpr int NU = G / 8;     // token n-tiles
    static constexpr int KU = G / 16;    // PV k-steps
    __host__ __device__ static constexpr int zn(bool dup) { return dup ? G / 8 : G / 4; }      // scores held per thread
};

template <int D, int G>
struct WarpState {
    using C = Cfg<D, G>;
    float o[C::MT][4];      // transposed output: channel rows (c0,c1) and their partners (c2,c3), head columns 2t, 2t+1; scaled 2^-16
    float ob[4];            // sum_j p_j * vlo[j][cg] for this thread's head (row r), cg = 2t, 2t+1 mod GV: hi (c0, c1) and lo (c2, c3); scaled 2^8
    float m;                // running reference of this thread's head (log2 domain), uniform over the quad
    float l;                // this thread's share of the running sum
};

template <int D, int G>
struct Ctx {                             // per-thread constants of the consumer role
    uint32_t qprep;                      // shared address of this lane's first prepared-query chunk (hi plane)
    float f;                             // 2^-eq * log2(e) of this thread's head
    int r, t, lane;
    bool part;                           // with head pairs in the rows: this thread feeds the lo column of its head
};

template <int D, int G>
__device__ __forceinline__ uint4 qchunk(const Ctx<D, G>& c, int plane, int i) {
    return lds_v4(c.qprep + (uint32_t)(plane * Cfg<D, G>::QPLANE * 2 + i * 512));
}

// Part of (ph + pl) * s that this thread's column carries: hi = rn(ph*s) with pm = pl = 0, or
// lo = rn(pl*s + (ph*s - hi)) with pm = -ph.
__device__ __forceinline__ uint32_t mul_part(uint32_t ph, uint32_t pm, uint32_t pl, uint32_t s) {
    const __half2 h = __hmul2(u32_as_h2(pm), u32_as_h2(s));
    const __half2 e = __hfma2(u32_as_h2(ph), u32_as_h2(s), h);
    return h2_as_u32(__hfma2(u32_as_h2(pl), u32_as_h2(s), e));
}

// klo or kstep pairs of the two k-steps of chunk i, in the arrangement of a rung's codes; `at` is the shared address of this
// thread's channels in the plane's group.
template <int D, int G, int BITS>
__device__ __forceinline__ void plane_pairs(uint32_t at, int i, uint32_t (&p)[4]) {
    if (BITS == 8) {
        const uint4 v = lds_v4(at + 16 * i);
        p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
    } else if (BITS == 4) {                              // s = 2x+y with x = i: words 4i+y, 4i+y+2
        const uint4 v = lds_v4(at + 16 * i);
        p[0] = prmt(v.x, v.z, 0x5410); p[1] = prmt(v.x, v.z, 0x7632);
        p[2] = prmt(v.y, v.w, 0x5410); p[3] = prmt(v.y, v.w, 0x7632);
    } else {                                             // s = 4x+y: x = i>>1, y = 2(i&1)+{0,1}: words 8x+y, 8x+y+4
        const uint32_t w0 = at + (uint32_t)(32 * (i >> 1) + 8 * (i & 1));
        const uint2 va = lds_v2(w0), vb = lds_v2(w0 + 16);
        p[0] = prmt(va.x, vb.x, 0x5410); p[1] = prmt(va.x, vb.x, 0x7632);
        p[2] = prmt(va.y, vb.y, 0x5410); p[3] = prmt(va.y, vb.y, 0x7632);
    }
}

// q . klo of every token group of a block in one n-tile: its eight columns are dealt to the groups (column n carries group
// n * TG / 8), so a block costs the MMAs of one group.  Returns the value of this thread's row's head (with head pairs: valid
// in odd rows) for the group of column 2t; unit_bias fetches a unit's.
template <int D, int G, int BITS, bool DUP>
__device__ __forceinline__ float block_bias(const Ctx<D, G>& c, uint32_t blk) {
    using C = Cfg<D, G>;
    constexpr int RB = D * BITS / 8;
    const uint32_t at = blk + (uint32_t)(2 * (kP * RB) + ((((c.r * C::TG) >> 3) * D + C::DT * c.t) * 2));
    float b0[4], b1[4];                                  // one per k-step of a chunk: independent MMAs
#pragma unroll
    for (int i = 0; i < C::CH; ++i) {
        uint32_t lp[4];
        plane_pairs<D, G, BITS>(at, i, lp);
        if (BITS == 4) {                                 // the query planes carry x16 on slots 0,1 (arr_scale): take it back out
            const __half2 k16 = __float2half2_rn(0.0625f);
            lp[0] = h2_as_u32(__hmul2(u32_as_h2(lp[0]), k16)); lp[2] = h2_as_u32(__hmul2(u32_as_h2(lp[2]), k16));
        } else if (BITS == 2) {                          // ... x4 on slots 2,3
            const __half2 k4 = __float2half2_rn(0.25f);
            lp[1] = h2_as_u32(__hmul2(u32_as_h2(lp[1]), k4)); lp[3] = h2_as_u32(__hmul2(u32_as_h2(lp[3]), k4));
        }
        uint4 qa, qb;
        if (DUP) {
            const uint4 h = qchunk(c, 0, i), l = qchunk(c, 2, i);
            qa = make_uint4(h.x, l.x, h.y, l.y); qb = make_uint4(h.z, l.z, h.w, l.w);
        } else {
            qa = qchunk(c, 0, i); qb = qchunk(c, 1, i);
        }
        if (i == 0) {
            mma_f16_z(b0, qa.x, qa.y, qa.z, qa.w, lp[0], lp[1]);
            mma_f16_z(b1, qb.x, qb.y, qb.z, qb.w, lp[2], lp[3]);
        } else {
            mma_f16(b0, qa.x, qa.y, qa.z, qa.w, lp[0], lp[1]);
            mma_f16(b1, qb.x, qb.y, qb.z, qb.w, lp[2], lp[3]);
        }
    }
    return (b0[0] + b0[2]) + (b1[0] + b1[2]);            // hi rows + lo rows, both k-steps
}
template <int D, int G, bool DUP>
__device__ __forceinline__ float unit_bias(const Ctx<D, G>& c, float b, int unit) {
    const int q = (unit * 4) / Cfg<D, G>::TG;
    return __shfl_sync(0xffffffffu, b, DUP ? (2 * c.t + 1) * 4 + q : (c.lane & 28) + q);
}

// ---- K side of one unit of a quantised block ---------------------------------------------------------
// Token octet n of the unit: its codes arrive as bb[n][0..3], the registers of k-steps 2i (0, 1) and 2i+1 (2, 3).
template <int D, int G, int BITS, int LW>
__device__ __forceinline__ void code_regs(const uint32_t (&W)[LW], int i, int ii, uint32_t (&b)[4]) {
    if (BITS == 8) {
        const uint32_t wx = W[(2 * ii) % LW], wy = W[(2 * ii + 1) % LW];
        b[0] = prmt(wx, 0u, 0x4140); b[1] = prmt(wx, 0u, 0x4342);
        b[2] = prmt(wy, 0u, 0x4140); b[3] = prmt(wy, 0u, 0x4342);
    } else if (BITS == 4) {
        const uint32_t w = W[ii % LW];
        const uint32_t u = rotl(w, 3), v = w >> 5;
        b[0] = u & 0x00780078u; b[1] = u & 0x07800780u;
        b[2] = v & 0x00780078u; b[3] = v & 0x07800780u;
    } else {
        // fields 4h..4h+3 (and +8) of the word, h = i & 1, brought to bits 8-9 / 6-7
        const uint32_t w = W[(ii >> 1) % LW] >> (8 * (ii & 1));
        const uint32_t u = rotl(w, 4);
        b[0] = rotl(w, 8) & 0x03000300u; b[1] = u & 0x00C000C0u;
        b[2] = u & 0x03000300u;          b[3] = w & 0x00C000C0u;
    }
}

// Scores of a unit, as multiples of k_unscale(BITS) * c.f above the unit's bias.
//
// Five to eight heads: S[head][token], the codes are the B operand; this thread holds its row's head and the tokens
// 8n + 2t, 8n + 2t + 1.  Up to four heads: S[token][head part], the codes are the A operand of half as many MMAs, whose eight
// columns are the (hi, lo) of every head; this thread holds head t and the tokens 8n + r.
template <int D, int G, int BITS, bool DUP>
__device__ __forceinline__ void scores_unit(const Ctx<D, G>& c, uint32_t blk, int tg, float (&z)[Unit<D, G>::zn(DUP)]) {
    using C = Cfg<D, G>;
    using UU = Unit<D, G>;
    constexpr int RB = D * BITS / 8;                     // bytes per token row
    constexpr int TB = RB / 4;                           // bytes per thread per row
    const uint32_t nat = blk + (uint32_t)(2 * (kP * RB) + C::KSCALE + (tg * D + C::DT * c.t) * 2);
    // The thread's codes of a token row are fetched with the widest load that fits (all chunks at
    // once for 4- and 2-bit codes): a quarter warp then reads whole rows side by side, free of the
    // bank conflicts that one 4-byte load per chunk had (rows are 32-128 bytes apart).
    constexpr int CB = TB / C::CH;                       // code bytes per thread, row and chunk
    constexpr int LB0 = TB < GKV_K_FETCH ? TB : GKV_K_FETCH;
    constexpr int LB = LB0 < CB ? CB : LB0;              // bytes per fetch (at least one chunk)
    constexpr int CG = LB / CB;                          // chunks per fetch
    constexpr int LW = LB / 4;
    static_assert(LB >= 4 && C::CH % CG == 0, "unsupported shape");
    // every fetch stays inside one 16-byte chunk, so in a swizzled block only the chunk moves (rows 8n + r of
    // all n-tiles have the same XOR term)
    static_assert(LB <= 16, "a fetch must not cross a 16-byte chunk");
    const uint32_t kx = swz_term<D, G, BITS>(c.r, 0);
    const uint32_t rowbase = blk + (uint32_t)((tg * UU::U + c.r) * RB);

    constexpr int NACC = DUP ? UU::NU / 2 : UU::NU;
    float acc[NACC][4];                                  // first written by the MMAs of chunk 0 (accumulator input zero)
#pragma unroll
    for (int g = 0; g < C::CH / CG; ++g) {
        uint32_t W[UU::NU][LW];
#pragma unroll
        for (int n = 0; n < UU::NU; ++n) {
            const uint32_t src = rowbase + (((uint32_t)(c.t * TB + g * LB)) ^ kx) + (uint32_t)(n * 8 * RB);
            if (LW == 4) { const uint4 v = lds_v4(src); W[n][0] = v.x; W[n][1 % LW] = v.y; W[n][2 % LW] = v.z; W[n][3 % LW] = v.w; }
            else if (LW == 2) { const uint2 v = lds_v2(src); W[n][0] = v.x; W[n][1 % LW] = v.y; }
            else W[n][0] = lds_u32(src);
        }
#pragma unroll
        for (int ii = 0; ii < CG; ++ii) {                // two k-steps at a time
            const int i = g * CG + ii;
            uint32_t sp[4];                              // kstep pairs of k-steps 2i and 2i+1 in this arrangement
            plane_pairs<D, G, BITS>(nat, i, sp);
            uint32_t bb[UU::NU][4];
#pragma unroll
            for (int n = 0; n < UU::NU; ++n) code_regs<D, G, BITS, LW>(W[n], i, ii, bb[n]);
            if (DUP) {
                const uint4 h = qchunk(c, 0, i), m = qchunk(c, 1, i), l = qchunk(c, 2, i);
                const uint32_t b0 = mul_part(h.x, m.x, l.x, sp[0]), b1 = mul_part(h.y, m.y, l.y, sp[1]);
                const uint32_t b2 = mul_part(h.z, m.z, l.z, sp[2]), b3 = mul_part(h.w, m.w, l.w, sp[3]);
#pragma unroll
                for (int n = 0; n < NACC; ++n) {
                    if (i == 0) mma_f16_z(acc[n], bb[2 * n][0], bb[2 * n + 1][0], bb[2 * n][1], bb[2 * n + 1][1], b0, b1);
                    else mma_f16(acc[n], bb[2 * n][0], bb[2 * n + 1][0], bb[2 * n][1], bb[2 * n + 1][1], b0, b1);
                }
#pragma unroll
                for (int n = 0; n < NACC; ++n)
                    mma_f16(acc[n], bb[2 * n][2], bb[2 * n + 1][2], bb[2 * n][3], bb[2 * n + 1][3], b2, b3);
            } else {
                const uint4 qa = qchunk(c, 0, i), qb = qchunk(c, 1, i);      // (hi, lo, hi, lo) of k-steps 2i and 2i+1
                uint32_t a[8];
                mul_split(qa.x, qa.y, sp[0], a[0], a[1]);
                mul_split(qa.z, qa.w, sp[1], a[2], a[3]);
                mul_split(qb.x, qb.y, sp[2], a[4], a[5]);
                mul_split(qb.z, qb.w, sp[3], a[6], a[7]);
                // k-step major: the two MMAs of an n-tile are NU issues apart, which hides the MMA latency
#pragma unroll
                for (int n = 0; n < NACC; ++n) {
                    if (i == 0) mma_f16_z(acc[n], a[0], a[1], a[2], a[3], bb[n][0], bb[n][1]);
                    else mma_f16(acc[n], a[0], a[1], a[2], a[3], bb[n][0], bb[n][1]);
                }
#pragma unroll
                for (int n = 0; n < NACC; ++n) mma_f16(acc[n], a[4], a[5], a[6], a[7], bb[n][2], bb[n][3]);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NACC; ++n) {
        z[2 * n + 0] = DUP ? acc[n][0] + acc[n][1] : acc[n][0] + acc[n][2];      // hi + lo
        z[2 * n + 1] = DUP ? acc[n][2] + acc[n][3] : acc[n][1] + acc[n][3];
    }
}

template <int D, int G, bool DUP>
__device__ __forceinline__ void scores_unit_bf16(const Ctx<D, G>& c, uint32_t blk, int tg, float (&z)[Unit<D, G>::zn(DUP)]) {
    using C = Cfg<D, G>;
    using UU = Unit<D, G>;
    // swizzled block: this thread's 16-byte chunks of a row all share the row's XOR term
    const uint32_t bt = (uint32_t)(C::DT * c.t * 2);
    const uint32_t kx = swz_term<D, G, 16>(c.r, (int)bt);
    const uint32_t rowbase = blk + (uint32_t)((tg * UU::U + c.r) * D * 2);
    constexpr int NACC = DUP ? UU::NU / 2 : UU::NU;
    float acc[NACC][4];
#pragma unroll
    for (int i = 0; i < C::CH; ++i) {
        uint4 w[UU::NU];
        const uint32_t coff = (bt + 16u * (uint32_t)i) ^ kx;
#pragma unroll
        for (int n = 0; n < UU::NU; ++n) w[n] = lds_v4(rowbase + coff + n * 8 * D * 2);
        if (DUP) {
            const uint4 b = qchunk(c, 0, i);
#pragma unroll
            for (int n = 0; n < NACC; ++n) {
                if (i == 0) mma_bf16_z(acc[n], w[2 * n].x, w[2 * n + 1].x, w[2 * n].y, w[2 * n + 1].y, b.x, b.y);
                else mma_bf16(acc[n], w[2 * n].x, w[2 * n + 1].x, w[2 * n].y, w[2 * n + 1].y, b.x, b.y);
            }
#pragma unroll
            for (int n = 0; n < NACC; ++n)
                mma_bf16(acc[n], w[2 * n].z, w[2 * n + 1].z, w[2 * n].w, w[2 * n + 1].w, b.z, b.w);
        } else {
            const uint4 qa = qchunk(c, 0, i), qb = qchunk(c, 1, i);
#pragma unroll
            for (int n = 0; n < NACC; ++n) {
                if (i == 0) mma_bf16_z(acc[n], qa.x, qa.y, qa.z, qa.w, w[n].x, w[n].y);
                else mma_bf16(acc[n], qa.x, qa.y, qa.z, qa.w, w[n].x, w[n].y);
            }
#pragma unroll
            for (int n = 0; n < NACC; ++n) mma_bf16(acc[n], qb.x, qb.y, qb.z, qb.w, w[n].z, w[n].w);
        }
    }
#pragma unroll
    for (int n = 0; n < NACC; ++n) {
        z[2 * n + 0] = DUP ? acc[n][0] + acc[n][1] : acc[n][0] + acc[n][2];
        z[2 * n + 1] = DUP ? acc[n][2] + acc[n][3] : acc[n][1] + acc[n][3];
    }
}

// ---- online-softmax update ---------------------------------------------------------------------
// The running reference m only moves when a score exceeds it by more than kLazy (log2 domain):
// until then weights are taken against the stale reference and may reach 2^kLazy.  That keeps
// the accumulator rescale off the common path; the fp16 weight operands still fit
// (p * 2^8 * step < 65504 for any step < 16).
constexpr float kLazy = 4.0f;
// Of 8- and 4-bit blocks the reference is a whole number: its sum with the weights' scale is exact, and their two halves have
// bits to spare below a largest weight of 1/2.  Raw values take the weights as two bf16 halves, 16 bits, of which a largest
// weight of exactly 1 needs one; 2-bit blocks' scale is 4, and what an octave lower would lose lies at the end of fp16's
// range.  Against whole numbers everywhere the error of raw blocks against 64 bits is 4.0e-6 of the result's norm instead of
// 4.6e-6 (500 tokens, 4.4e-6 and 4.9e-6 at 2000), that of 2-bit blocks 1 to 10 % lower.
__host__ __device__ constexpr bool whole_reference(int wscale) { return wscale >= 5; }

// The accumulators are indexed by head COLUMN (2t, 2t+1) while the reference belongs to the head of
// the thread's ROW, so the rescale factors of the two columns come from the lanes that own them.
template <int D, int G, bool DUP, bool WHOLE>
__device__ __forceinline__ float move_reference(const Ctx<D, G>& c, WarpState<D, G>& st, float mx) {
    using C = Cfg<D, G>;
    const bool need = mx > st.m + kLazy || st.m == -INFINITY;   // per head (uniform over the quad)
    if (__any_sync(0xffffffffu, need)) {
        const float mnew = need ? (WHOLE ? ceilf(mx) : mx) : st.m;
        const float corr = ex2(st.m - mnew);          // 0 when st.m = -inf, 1 for the heads that stay
        st.m = mnew;
        st.l *= corr;
        // With head pairs this thread's reference and both its columns belong to head t, and the p . vlo rows to head r / 2
        // (lane r / 2 of the first row has it).  Otherwise its columns are the heads 2t and 2t+1, whose references are in the
        // rows of those numbers.
        const float c0 = DUP ? corr : __shfl_sync(0xffffffffu, corr, 8 * c.t);
        const float c1 = DUP ? corr : __shfl_sync(0xffffffffu, corr, 8 * c.t + 4);
        const float cb = DUP ? __shfl_sync(0xffffffffu, corr, c.r >> 1) : corr;
#pragma unroll
        for (int n = 0; n < C::MT; ++n) {
            st.o[n][0] *= c0; st.o[n][1] *= c1; st.o[n][2] *= c0; st.o[n][3] *= c1;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) st.ob[i] *= cb;
    }
    return st.m;
}

// z: scores of this thread's head for its tokens of the unit, as multiples of `scale` above `bias` (log2
// domain); nrel = valid tokens left in this unit (>= 1).  Returns the weights times 2^PS in z: the two scales, the reference
// and the power of two the value product wants are one fused multiply-add per score.
template <int D, int G, bool DUP, int PS>
__device__ __forceinline__ float softmax_unit(const Ctx<D, G>& c, WarpState<D, G>& st, float (&z)[Unit<D, G>::zn(DUP)], float scale, float bias, int nrel) {
    using UU = Unit<D, G>;
    constexpr int ZN = UU::zn(DUP);
    float mx = -INFINITY;
    if (nrel >= UU::U) {                                 // full unit (the common case): no masks
#pragma unroll
        for (int i = 0; i < ZN; ++i) mx = fmaxf(mx, z[i]);
    } else {
#pragma unroll
        for (int i = 0; i < ZN; ++i) {
            const int tok = DUP ? 8 * i + c.r : (i >> 1) * 8 + 2 * c.t + (i & 1);
            if (tok >= nrel) z[i] = -INFINITY;
            mx = fmaxf(mx, z[i]);
        }
    }
    mx = fmaf(mx, scale, bias);
#pragma unroll
    for (int o = DUP ? 4 : 1; o < (DUP ? 32 : 4); o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float m = move_reference<D, G, DUP, whole_reference(PS)>(c, st, mx);
    const float shift = bias - (m - (float)PS);
    float ls = 0.f;
#pragma unroll
    for (int i = 0; i < ZN; ++i) {
        z[i] = ex2(fmaf(z[i], scale, shift));
        ls += z[i];
    }
    st.l += ls;
    return ls;                                           // this thread's share of the unit's weights (reference st.m), times 2^PS
}

// Pairs (x[tok][cg], x[tok+1][cg]) of a (64, GV) fp16 plane at shared address `row` (token `tok`, even).
template <int GV>
__device__ __forceinline__ void scale_pairs(uint32_t row, uint32_t (&out)[GV]) {
    if (GV == 8) {
        const uint4 a = lds_v4(row), b = lds_v4(row + 16);
        out[0] = prmt(a.x, b.x, 0x5410); out[1 % GV] = prmt(a.x, b.x, 0x7632);
        out[2 % GV] = prmt(a.y, b.y, 0x5410); out[3 % GV] = prmt(a.y, b.y, 0x7632);
        out[4 % GV] = prmt(a.z, b.z, 0x5410); out[5 % GV] = prmt(a.z, b.z, 0x7632);
        out[6 % GV] = prmt(a.w, b.w, 0x5410); out[7 % GV] = prmt(a.w, b.w, 0x7632);
    } else if (GV == 4) {
        const uint4 v = lds_v4(row);
        out[0] = prmt(v.x, v.z, 0x5410); out[1 % GV] = prmt(v.x, v.z, 0x7632);
        out[2 % GV] = prmt(v.y, v.w, 0x5410); out[3 % GV] = prmt(v.y, v.w, 0x7632);
    } else if (GV == 2) {
        const uint2 v = lds_v2(row);
        out[0] = prmt(v.x, v.y, 0x5410); out[1 % GV] = prmt(v.x, v.y, 0x7632);
    } else {
#pragma unroll
        for (int cg = 0; cg < GV; ++cg) out[cg] = lds_u16(row + 2 * cg) | (lds_u16(row + 2 * GV + 2 * cg) << 16);
    }
}

// ---- V side: the transposed product O^T[channel][head] += V^T[channel][token] * (p*vstep)[token][head] -------
// How a thread's value codes reach its A registers.  A SPAN is the set of channels whose codes one
// fetch delivers: the 16-byte chunk of a token row that ldmatrix.trans hands out (128/BITS channels;
// used for 8-bit codes, and for 4-bit codes when a channel group is at least a chunk), or one
// channel group fetched with a plain byte load (2-bit codes, and 4-bit codes with 16-channel groups).
// Either way thread r owns F = SP/8 neighbouring fields of every span, fields 2k and 2k+1 feed rows r
// and r+8 of the span's m-tile k, and the register R = {fields of token a | fields of token a+1 << 16}
// is unpacked by one shift and two masks per m-tile: the even field lands on bit POS, the odd one
// BITS higher, so rows r+8 carry 2^BITS more weight, which the epilogue takes back out.
template <int D, int G, int BITS>
struct VT {
    static constexpr bool LDSM = BITS == 8 || (BITS == 4 && G >= 32);
    static constexpr int SP = LDSM ? 128 / BITS : G;     // channels per span
    static constexpr int F = SP / 8;                     // fields per thread and span
    static constexpr int MTS = F / 2;                    // m-tiles per span
    static constexpr int SPC = G / SP;                   // spans per channel group
    static constexpr int NSPAN = D / SP;
    static constexpr int RB = D * BITS / 8;
    static constexpr int POS = BITS == 4 ? 3 : BITS == 2 ? 6 : 0;
    static constexpr int LOAD_BITS = F * BITS;           // bits of one token a thread needs per span (plain-load path)
    static_assert(F >= 2 && F % 2 == 0 && SPC >= 1, "unsupported shape");
};
// log2 of the scale the weights carry: 2^(8-POS) for codes, 2^-16 for raw values (the same accumulator scale)
__host__ __device__ constexpr int v_wscale(int bits) { return bits == 16 ? -16 : bits == 4 ? 5 : bits == 2 ? 2 : 8; }
__host__ __device__ constexpr float pow2(int e) { return e >= 0 ? (float)(1 << e) : 1.f / (float)(1 << -e); }
__host__ __device__ constexpr float v_rowscale(int bits) { return bits == 4 ? 16.f : bits == 2 ? 4.f : 1.f; }   // weight of rows r+8 over rows r

// A registers (rows r, r+8) of m-tile k of a span from R (the thread's first field at bit 0 of each half).
template <int BITS, int POS>
__device__ __forceinline__ void extract_pair(uint32_t R, int k, uint32_t& even, uint32_t& odd) {
    if (BITS == 8) {
        even = prmt(R, 0u, 0x4240);
        odd = prmt(R, 0u, 0x4341);
    } else {
        constexpr uint32_t FM = (1u << BITS) - 1u;
        const int sh = POS - 2 * k * BITS;
        const uint32_t u = sh >= 0 ? rotl(R, sh) : (R >> (-sh));
        even = u & ((FM << POS) * 0x00010001u);
        odd = u & ((FM << (POS + BITS)) * 0x00010001u);
    }
}

// Up to four heads: the weights of head t for the tokens r (x0) and r + 8 (x1) of a k-step become the columns of the value
// product: column r is the hi (even) or lo half of head r / 2, a register holds the tokens 2t, 2t+1 of the first or second
// half of the k-step.  The 8x8 transposition is one movmatrix per register.
//   codes (RAW = false): h = the hi halves in every column, l = the lo halves in the lo columns, m = -hi there, else 0;
//   raw values: h = the column's own half.
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
template <bool RAW, class CtxT>
__device__ __forceinline__ void head_columns(const CtxT& c, float x0, float x1, uint32_t (&h)[2], uint32_t (&l)[2], uint32_t (&m)[2]) {
    uint32_t hi, lo;
    if (RAW) {
        split_bf16x2(x0, x1, hi, lo);
        h[0] = transpose8(prmt(hi, lo, 0x5410));
        h[1] = transpose8(prmt(hi, lo, 0x7632));
    } else {
        split_f16x2(x0, x1, hi, lo);
        h[0] = transpose8(prmt(hi, hi, 0x5410));
        h[1] = transpose8(prmt(hi, hi, 0x7632));
        l[0] = transpose8(lo << 16);
        l[1] = transpose8(lo & 0xffff0000u);
        const uint32_t on = c.part ? 0xffffffffu : 0u;
        m[0] = (h[0] ^ 0x80008000u) & on;
        m[1] = (h[1] ^ 0x80008000u) & on;
    }
}

template <int D, int G, int BITS, bool DUP>
__device__ __forceinline__ void values_unit(const Ctx<D, G>& c, WarpState<D, G>& st, uint32_t blk, int unit,
                                            const float (&pz)[Unit<D, G>::zn(DUP)]) {
    using C = Cfg<D, G>;
    using UU = Unit<D, G>;
    using V = VT<D, G, BITS>;
    constexpr int RB = V::RB;
    const uint32_t vbase = blk + (uint32_t)(kP * RB);
    const uint32_t sbase = blk + (uint32_t)(2 * (kP * RB) + 2 * C::KSCALE);       // vlo plane; vstep follows
    const int tok0 = unit * UU::U + 2 * c.t;            // lower token of this thread's first pair
    // ldmatrix row of this lane: token (lane & 7) of the first or second half of a k-step, chunk +0 / +1; in a
    // swizzled block the chunk index is XORed with the row's term (the same for every row this lane addresses)
    const uint32_t vx = swz_term<D, G, BITS>(c.lane & 7, 0);
    const uint32_t ldsm_lane = vbase + (uint32_t)((unit * UU::U + (c.lane & 7) + 8 * ((c.lane >> 3) & 1)) * RB) +
                               ((uint32_t)(16 * (c.lane >> 4)) ^ (vx & 16u));
    const uint32_t vxe = vx & ~16u;
    // plain-load path: this thread's fields of (token tok0, span 0)
    const uint32_t lds_lane = vbase + (uint32_t)(tok0 * RB + (c.r * V::LOAD_BITS) / 8);
    const int sub = (V::LOAD_BITS % 8) ? ((c.r * V::LOAD_BITS) & 7) : 0;
    const int cgr = c.r % C::GV;
#pragma unroll
    for (int ku = 0; ku < UU::KU; ++ku) {
        uint32_t ph[2], pl[2], pm[2];                    // with head pairs: the operands of mul_part
        if (DUP) head_columns<false>(c, pz[(2 * ku) % UU::zn(DUP)], pz[(2 * ku + 1) % UU::zn(DUP)], ph, pl, pm);
        else {
            split_f16x2(pz[(4 * ku + 0) % UU::zn(DUP)], pz[(4 * ku + 1) % UU::zn(DUP)], ph[0], pl[0]);
            split_f16x2(pz[(4 * ku + 2) % UU::zn(DUP)], pz[(4 * ku + 3) % UU::zn(DUP)], ph[1], pl[1]);
        }
        const uint32_t srow = sbase + (uint32_t)((tok0 + 16 * ku) * C::GV * 2);
        uint32_t sa[C::GV], sb[C::GV];
        scale_pairs<C::GV>(srow + C::VSCALE, sa);                      // vstep of the pair in n-tile 2ku
        scale_pairs<C::GV>(srow + C::VSCALE + 8 * C::GV * 2, sb);      // ... and of the pair in n-tile 2ku+1
        // p . vlo: heads are the rows (hi, lo), column n is channel group n mod GV
        {
            uint32_t la = lds_u16(srow + 2 * cgr) | (lds_u16(srow + 2 * C::GV + 2 * cgr) << 16);
            uint32_t lb = lds_u16(srow + 16 * C::GV + 2 * cgr) | (lds_u16(srow + 18 * C::GV + 2 * cgr) << 16);
            if (V::POS) {                               // keep the 2^8 scale of the p . vlo accumulator
                const __half2 lo_scale = __float2half2_rn((float)(1 << V::POS));
                la = h2_as_u32(__hmul2(u32_as_h2(la), lo_scale));
                lb = h2_as_u32(__hmul2(u32_as_h2(lb), lo_scale));
            }
            // The tensor core truncates: sums of one sign, as this one and that of the codes it is added to, drift towards zero
            // with every addition, and the two drifts cancel where both take the same number of additions.  With five to
            // eight heads an output takes two per k-step (hi and lo).  8-bit codes, 1M tokens, eight heads: error against 64
            // bits 1.3e-4 of the result's norm with one addition here, 4.7e-5 with two.  Products of narrow codes are short
            // enough that most of their additions are exact: there one is nearer (4 bits 1.5e-4 against 3.0e-4, 2 bits 2.3e-4
            // against 3.5e-4).
            if (BITS == 8 && !DUP) {
                mma_f16(st.ob, ph[0], 0u, ph[1], 0u, la, lb);
                mma_f16(st.ob, pl[0], 0u, pl[1], 0u, la, lb);
            } else {
                mma_f16(st.ob, ph[0], pl[0], ph[1], pl[1], la, lb);
            }
        }
        // value codes of this k-step: Rlo[s] / Rhi[s] = span s, token pairs of n-tiles 2ku / 2ku+1
        uint32_t Rlo[V::NSPAN], Rhi[V::NSPAN];
        if (V::LDSM) {
#pragma unroll
            for (int s2 = 0; s2 < V::NSPAN / 2; ++s2)
                ldsm_x4_trans(ldsm_lane + (uint32_t)(ku * 16 * RB) + ((uint32_t)(32 * s2) ^ vxe), Rlo[2 * s2], Rhi[2 * s2],
                              Rlo[(2 * s2 + 1) % V::NSPAN], Rhi[(2 * s2 + 1) % V::NSPAN]);
        } else {
#pragma unroll
            for (int s = 0; s < V::NSPAN; ++s) {
                uint32_t x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t src = lds_lane + (uint32_t)((16 * ku + ((k & 2) ? 8 : 0) + (k & 1)) * RB + (s * V::SP * BITS) / 8);
                    x[k] = V::LOAD_BITS > 8 ? lds_u16(src) : (lds_u8(src) >> sub);
                }
                Rlo[s] = prmt(x[0], x[1], 0x5410);
                Rhi[s] = prmt(x[2], x[3], 0x5410);
            }
        }
#pragma unroll
        for (int cg = 0; cg < C::GV; ++cg) {
            uint32_t b0h, b0l, b1h, b1l;
            if (DUP) {
                b0h = mul_part(ph[0], pm[0], pl[0], sa[cg]);
                b1h = mul_part(ph[1], pm[1], pl[1], sb[cg]);
                b0l = b1l = 0u;
            } else {
                mul_split(ph[0], pl[0], sa[cg], b0h, b0l);
                mul_split(ph[1], pl[1], sb[cg], b1h, b1l);
            }
#pragma unroll
            for (int sc = 0; sc < V::SPC; ++sc) {
                const int s = cg * V::SPC + sc;
#pragma unroll
                for (int k = 0; k < V::MTS; ++k) {
                    uint32_t a0, a1, a2, a3;
                    extract_pair<BITS, V::POS>(Rlo[s], k, a0, a1);
                    extract_pair<BITS, V::POS>(Rhi[s], k, a2, a3);
                    float (&acc)[4] = st.o[s * V::MTS + k];
                    mma_f16(acc, a0, a1, a2, a3, b0h, b1h);
                    if (!DUP) mma_f16(acc, a0, a1, a2, a3, b0l, b1l);
                }
            }
        }
    }
}

// Raw bf16 values: m-tile m is channels 16m .. 16m+15 in natural order; ldmatrix.trans delivers the
// four A registers of a (k-step, m-tile) directly.
template <int D, int G, bool DUP>
__device__ __forceinline__ void values_unit_bf16(const Ctx<D, G>& c, WarpState<D, G>& st, uint32_t blk, int unit,
                                                 const float (&pz)[Unit<D, G>::zn(DUP)]) {
    using C = Cfg<D, G>;
    using UU = Unit<D, G>;
    constexpr int RB = D * 2;
    // matrices: (tokens of n-tile 2ku, channels 16m..), (same tokens, 16m+8..), (n-tile 2ku+1, 16m..), (n-tile 2ku+1, 16m+8..)
    // swizzled: chunk (2m + b) of a row, b = (lane >> 3) & 1, is XORed with the term of its 128-byte tile row
    const uint32_t rowb = blk + (uint32_t)(kP * RB + (unit * UU::U + (c.lane & 7) + 8 * (c.lane >> 4)) * RB);
    const uint32_t cb = 16u * ((c.lane >> 3) & 1);
    const uint32_t vx0 = swz_term<D, G, 16>(c.lane & 7, 0), vx1 = swz_term<D, G, 16>(c.lane & 7, 128);   // first / second 128 bytes of the row
#pragma unroll
    for (int ku = 0; ku < UU::KU; ++ku) {
        uint32_t b0, b1, l0 = 0u, l1 = 0u;               // with head pairs the columns hold both halves
        if (DUP) {
            uint32_t own[2], none[2], pm[2];
            head_columns<true>(c, pz[(2 * ku) % UU::zn(DUP)], pz[(2 * ku + 1) % UU::zn(DUP)], own, none, pm);
            b0 = own[0]; b1 = own[1];
        } else {
            split_bf16x2(pz[(4 * ku + 0) % UU::zn(DUP)], pz[(4 * ku + 1) % UU::zn(DUP)], b0, l0);
            split_bf16x2(pz[(4 * ku + 2) % UU::zn(DUP)], pz[(4 * ku + 3) % UU::zn(DUP)], b1, l1);
        }
#pragma unroll
        for (int m = 0; m < C::MT; ++m) {
            uint32_t a0, a1, a2, a3;
            const uint32_t off = (uint32_t)(32 * m) + cb;                 // byte of the chunk inside the row
            const uint32_t phys = (32 * m >= 128) ? (off ^ vx1) : (off ^ vx0);
            ldsm_x4_trans(rowb + (uint32_t)(ku * 16 * RB) + phys, a0, a1, a2, a3);
            mma_bf16(st.o[m], a0, a1, a2, a3, b0, b1);
            if (!DUP) mma_bf16(st.o[m], a0, a1, a2, a3, l0, l1);
        }
    }
}

// A block whose tail is not valid: clear what the value product would otherwise read for the
// tokens beyond nvalid (those bytes may hold anything, even NaN patterns), so that the main
// path needs no masks.  Scores of such tokens are forced to -inf by the softmax.
template <int D, int G>
__device__ __forceinline__ void clear_invalid_tail(uint8_t* blk, int level, int nvalid, int lane) {
    using C = Cfg<D, G>;
    if (level == 16) {
        uint32_t* v = reinterpret_cast<uint32_t*>(blk + kP * D * 2 + nvalid * D * 2);
        for (int i = lane; i < (kP - nvalid) * D / 2; i += 32) v[i] = 0u;
    } else {
        const int RB = D * level / 8;
        uint16_t* lo = reinterpret_cast<uint16_t*>(blk + 2 * kP * RB + 2 * C::KSCALE);
        for (int i = nvalid * C::GV + lane; i < kP * C::GV; i += 32) { lo[i] = 0; lo[C::VSCALE / 2 + i] = 0; }
    }
    fence_before_bulk();        // the next copy into these bytes comes from the producer, after the pair has released them
    __syncwarp();
}

// F neighbouring floats of a record's o row (F = 2, 4 or 8; the row starts on 16 bytes).
template <int F>
__device__ __forceinline__ void store_run(float* dst, const float (&x)[F]) {
    if (F == 2) *reinterpret_cast<float2*>(dst) = make_float2(x[0], x[1]);
    else {
#pragma unroll
        for (int i = 0; i < F; i += 4)
            *reinterpret_cast<float4*>(dst + i) = make_float4(x[i], x[(i + 1) % F], x[(i + 2) % F], x[(i + 3) % F]);
    }
}

// This warp's record of an item (natural-log domain): (m, l) and o[D] per head.
//
// A thread's channels of a span are F neighbours (channel SP * s + F * r + field), so they go out as one run; one
// float at a time, every store touched 32 sectors, eight times what the bytes need.
template <int D, int G, int BITS, bool DUP>
__device__ __forceinline__ void write_record(const Params& p, const Ctx<D, G>& c, const WarpState<D, G>& st, size_t rec0) {
    using C = Cfg<D, G>;
    float l = st.l;
#pragma unroll
    for (int o = DUP ? 4 : 1; o < (DUP ? 32 : 4); o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const int myhead = DUP ? c.t : c.r;
    if ((DUP ? c.r : c.t) == 0 && myhead < p.rep)
        p.part_ml[rec0 + myhead] = make_float2(st.m * 0.6931471805599453f, l * pow2(-v_wscale(BITS)));
    constexpr float kRow = 65536.f, kRow8 = 65536.f / v_rowscale(BITS);
    // heads of this thread's columns: t when the columns 2t, 2t+1 are its hi and lo halves, else 2t and 2t+1
    const int h0 = DUP ? c.t : 2 * c.t;
    float* out0 = p.part + (rec0 + h0) * D;
    float* out1 = out0 + D;
    const bool has0 = h0 < p.rep, has1 = !DUP && h0 + 1 < p.rep;
    if (BITS == 16) {
        // channels 16 m + r and 16 m + 8 + r: eight lanes fill a 32-byte sector
#pragma unroll
        for (int mt = 0; mt < C::MT; ++mt) {
            const float (&o)[4] = st.o[mt];
            const int ch = 16 * mt + c.r;
            if (has0) { out0[ch] = (DUP ? o[0] + o[1] : o[0]) * kRow; out0[ch + 8] = (DUP ? o[2] + o[3] : o[2]) * kRow; }
            if (has1) { out1[ch] = o[1] * kRow; out1[ch + 8] = o[3] * kRow; }
        }
    } else {
        using V = VT<D, G, BITS == 16 ? 8 : BITS>;
        // p . vlo of a head and channel group cg sits in the head's row, quad position cg / 2, element cg mod 2, scaled 2^8
        const float ob[2] = {st.ob[0] + st.ob[2], st.ob[1] + st.ob[3]};
        const int row0 = (DUP ? 2 * h0 + 1 : h0) * 4;                 // with head pairs the odd row has both halves
#pragma unroll
        for (int s = 0; s < V::NSPAN; ++s) {
            constexpr float kLo = 0.00390625f;
            const int cg = s / V::SPC;                                  // a span lies in one channel group
            const float bias0 = __shfl_sync(0xffffffffu, ob[cg & 1], row0 + (cg >> 1)) * kLo;
            const float bias1 = DUP ? 0.f : __shfl_sync(0xffffffffu, ob[cg & 1], row0 + 4 + (cg >> 1)) * kLo;
            float x0[V::F], x1[V::F];
#pragma unroll
            for (int k = 0; k < V::MTS; ++k) {
                const float (&o)[4] = st.o[s * V::MTS + k];
                x0[2 * k] = fmaf(DUP ? o[0] + o[1] : o[0], kRow, bias0);
                x0[2 * k + 1] = fmaf(DUP ? o[2] + o[3] : o[2], kRow8, bias0);
                x1[2 * k] = fmaf(o[1], kRow, bias1);
                x1[2 * k + 1] = fmaf(o[3], kRow8, bias1);
            }
            const int ch = V::SP * s + V::F * c.r;
            if (has0) store_run<V::F>(out0 + ch, x0);
            if (has1) store_run<V::F>(out1 + ch, x1);
        }
    }
}

// One thread per head and unit reports the head's share of a block's softmax mass: the reference in use
// (natural-log domain) and the sum of the unit's weights against it.
template <int D, int G, bool DUP>
__device__ __forceinline__ void report_mass(const Params& p, const Ctx<D, G>& c, int row, int orig, int upb, int unit, float ref, float sum) {
    const int head = DUP ? c.t : c.r;
    if ((DUP ? c.r : c.t) == 0 && head < p.rep)
        p.mass_part[(((size_t)row * p.nb + orig) * upb + unit) * p.rep + head] = make_float2(ref, sum);
}

// A narrow block is one warp's work, a wide one is shared by the two warps of a pair (a unit or two each).  A block per warp
// halves what a block costs besides its units (32 x 16k tokens at 4 bits, four heads per row 185 -> 165 us, eight 216 -> 202),
// but twelve blocks are being read at a time, which the rings hold with room for what comes next up to kSoloBytes; and an
// item of fewer than four rounds of blocks ends sooner when two warps share each (one sequence of 1000 tokens, items of six
// blocks: 13.5 against 13.1 us from a graph).
constexpr int kSoloBytes = 12288;
constexpr int kSoloBlocks = 24;
template <int D, int G, int BITS>
struct Share {
    static constexpr bool SOLO = BITS != 16 && 2 * kP * D * BITS / 8 + 4 * Cfg<D, G>::KSCALE <= kSoloBytes;
};

// An item of one of the byte-ring rungs: this warp's blocks of its stream (which begin at position `beg`), then its record.
template <int D, int G, int BITS, bool DUP, bool MASS>
__device__ __forceinline__ int ring_item(const Params& p, Smem<D, G>& sm, const Ctx<D, G>& c, const ItemDesc& it, int stream,
                                         int pair, int half, int beg, int end, size_t rec0) {
    using C = Cfg<D, G>;
    using UU = Unit<D, G>;
    using SH = Share<D, G, BITS>;
    constexpr int QB = BITS == 16 ? 8 : BITS;
    constexpr int UPB = kP / UU::U;                 // units per block; a pair's second warp has none of a block with a single one
    const bool solo = SH::SOLO && it.nblk >= kSoloBlocks;
    const int u0 = solo || UPB < 2 ? 0 : half * (UPB / 2);
    const int u1 = solo ? UPB : UPB >= 2 ? u0 + UPB / 2 : (half == 0 ? 1 : 0);
    WarpState<D, G> st;
#pragma unroll
    for (int n = 0; n < C::MT; ++n) st.o[n][0] = st.o[n][1] = st.o[n][2] = st.o[n][3] = 0.f;
    st.ob[0] = st.ob[1] = st.ob[2] = st.ob[3] = 0.f;
    st.m = -INFINITY;
    st.l = 0.f;
    const uint32_t ring = smem_u32(sm.ring) + (uint32_t)stream * kRingBytes;
    uint64_t* full = sm.full + stream * kNSlot;
    uint64_t* empty = sm.empty + stream * kNSlot;
    const Desc* desc = sm.desc + stream * kNSlot;
    const float scale = BITS == 16 ? c.f : k_unscale(QB) * c.f;
    // blocks are dealt by their position in the stream, across items
    const int mine = solo ? 2 * pair + half : pair;
    const int step = solo ? 2 * kPairsPerStream : kPairsPerStream;       // warps, or pairs, that take the stream's blocks in turn
    for (int seq = beg + (mine + step - beg % step) % step; seq < end; seq += step) {
        const int slot = seq % kNSlot;
        if (!mbar_wait(&full[slot], (uint32_t)(seq / kNSlot) & 1u)) return 4;
        const uint32_t off = desc[slot].off;
        const int nvalid = desc[slot].nvalid;
        const int orig = MASS ? desc[slot].orig : 0;
        const uint32_t blk = ring + off;
        // both warps of a pair clear the tail (same zeros, so the overlap is harmless)
        if (nvalid < kP) clear_invalid_tail<D, G>(sm.ring + (size_t)stream * kRingBytes + off, BITS, nvalid, c.lane);
        float bias_all = 0.f;
        if (BITS != 16 && u0 < u1) bias_all = block_bias<D, G, QB, DUP>(c, blk);
#pragma unroll 1
        for (int unit = u0; unit < u1; ++unit) {
            const int nrel = nvalid - unit * UU::U;
            if (nrel <= 0) {                             // no valid token in this unit: it weighs nothing
                if (MASS) report_mass<D, G, DUP>(p, c, it.row, orig, UPB, unit, -INFINITY, 0.f);
                if (MASS) continue;
                break;
            }
            float z[UU::zn(DUP)];
            if (BITS == 16) scores_unit_bf16<D, G, DUP>(c, blk, unit, z);
            else scores_unit<D, G, QB, DUP>(c, blk, unit, z);
            const float bias = BITS == 16 ? 0.f : unit_bias<D, G, DUP>(c, bias_all, unit) * c.f;
            float ls = softmax_unit<D, G, DUP, v_wscale(BITS)>(c, st, z, scale, bias, nrel);
            if (MASS) {
#pragma unroll
                for (int o = DUP ? 4 : 1; o < (DUP ? 32 : 4); o <<= 1) ls += __shfl_xor_sync(0xffffffffu, ls, o);
                report_mass<D, G, DUP>(p, c, it.row, orig, UPB, unit, st.m * 0.6931471805599453f, ls * pow2(-v_wscale(BITS)));
            }
            if (BITS == 16) values_unit_bf16<D, G, DUP>(c, st, blk, unit, z);
            else values_unit<D, G, QB, DUP>(c, st, blk, unit, z);
        }
        __syncwarp();
        if (c.lane == 0) mbar_arrive_n(&empty[slot], solo ? 2 : 1);      // the slot expects a pair
    }
    write_record<D, G, BITS, DUP>(p, c, st, rec0);
    return 0;
}

// Sixteen bytes of a cache row, which may stand at any address.
__device__ __forceinline__ uint4 ldg16(const uint8_t* src) {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) return __ldg(reinterpret_cast<const uint4*>(src));
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = (uint32_t)src[4 * i] | ((uint32_t)src[4 * i + 1] << 8) | ((uint32_t)src[4 * i + 2] << 16) | ((uint32_t)src[4 * i + 3] << 24);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// An item of centroid blocks: one key and one value vector stand for nvalid tokens (512 bytes per block at D = 128).  No
// ring: a warp takes TILES of sixteen blocks and treats them as sixteen tokens of fp16 rows whose weights are multiplied by
// the blocks' counts.  The fragments of both products come straight from global memory: a thread's keys are its quad
// position's channels of the tokens r and r + 8 (the B operand of S[head][token], query halves in rows 0-7 and 8-15), its
// values D / 8 neighbouring channels of the tokens 2t, 2t+1, 2t+8, 2t+9, paired up by one permutation per register (the B
// operand of O[head][channel], weight halves in the rows).  So O's columns 2t and 2t+1 of this thread are the D / 4 channels
// from t * D / 4, whole runs of its record.
//
// Both operands are two fp16 halves of 22 bits; what is added up stays in fp32 and is rounded, not truncated: every MMA starts
// from zero and its result is added by the FP32 pipes (sixteen blocks at a time that costs nothing: 42.3 us for 128 x 16k
// tokens of eight heads per row with and without), and scores, reference and record are in natural units, a power of two
// away from the products.  Against 64 bits the error of a row of centroids alone is that of FP32 arithmetic throughout: 1.2e-7
// of the result's norm at 2000 and at 16k tokens, 2.0e-7 where a few tokens dominate; sums kept in the MMAs' accumulators
// and scores in units of log2: 2.5e-7 at 2000 tokens, 4.5e-7 where a few dominate.
//
// On the FP32 pipes, a block at a time with a shuffle reduction per head, a block took a warp 4200 cycles, as much as one of
// 64 tokens at 4 bits.  32 x 16k tokens, all centroids, four heads per row 62 -> 35 us; 128 x 16k, two rows of eight heads
// 78 -> 42; 256 ragged sequences demoted to 4 bits 404 -> 338 with the other changes of that time, 343 before the sums
// left the accumulators.
template <int D, int G, bool MASS>
__device__ __forceinline__ void centroid_item(const Params& p, const Ctx<D, G>& c, const ItemDesc& it, const uint4* tab,
                                              int first, float qscale, size_t rec0) {
    using C = Cfg<D, G>;
    constexpr int NK = C::DT / 8;                         // 16-byte pieces of this thread's key channels
    constexpr int VC = D / 8, NV = VC / 8;                // its value channels per token, and their 16-byte pieces
    constexpr float kScale = 256.f;                       // weights are at most 64: well inside fp16, and far from its subnormals
    const int tiles = (it.nblk + 15) >> 4;
    const float unscale = 1.0f / qscale;                  // a power of two
    float o[VC][2];
#pragma unroll
    for (int i = 0; i < VC; ++i) o[i][0] = o[i][1] = 0.f;
    float m = -INFINITY, l = 0.f;                         // natural-log domain
    for (int tile = first; tile < tiles; tile += kConsumerWarps) {
        const int b0 = tile * 16;
        // entries beyond the item repeat its last one; their scores are masked
        auto entry = [&](int i) { return tab[min(b0 + i, it.nblk - 1)]; };
        auto source = [&](const uint4& e) { return p.data + (((unsigned long long)e.y << 32) | e.x); };
        // the values come after the scores are known (registers); until then they move as far as L2
        if (2 * D >= 128 * (c.lane >> 4) + 128) prefetch_l2(source(entry(c.lane & 15)) + 2 * D + 128 * (c.lane >> 4));
        uint4 kw[2][NK];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint8_t* src = source(entry(c.r + 8 * j)) + 2 * C::DT * c.t;
#pragma unroll
            for (int i = 0; i < NK; ++i) kw[j][i] = ldg16(src + 16 * i);
        }
        float cnt[4];
        int orig[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = 2 * c.t + (j & 1) + 8 * (j >> 1);
            const uint4 e = entry(i);
            cnt[j] = b0 + i < it.nblk ? (float)((e.z >> 8) & 0xffu) : 0.f;
            orig[j] = (int)e.w;
        }
        float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < C::CH; ++i) {
            const uint4 qa = qchunk(c, 0, i), qb = qchunk(c, 1, i);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint4 w = kw[j][i % NK];
                float a[4], b[4];
                mma_f16_z(a, qa.x, qa.y, qa.z, qa.w, w.x, w.y);
                mma_f16_z(b, qb.x, qb.y, qb.z, qb.w, w.z, w.w);
                z[2 * j] += (a[0] + b[0]) + (a[2] + b[2]);
                z[2 * j + 1] += (a[1] + b[1]) + (a[3] + b[3]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) z[j] = cnt[j] > 0.f ? z[j] * unscale : -INFINITY;
        uint4 vw[4][NV];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint8_t* src = source(entry(2 * c.t + (j & 1) + 8 * (j >> 1))) + 2 * D + 2 * VC * c.r;
#pragma unroll
            for (int h = 0; h < NV; ++h) vw[j][h] = ldg16(src + 16 * h);
        }
        float mx = fmaxf(fmaxf(z[0], z[1]), fmaxf(z[2], z[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        if (__any_sync(0xffffffffu, mx > m)) {
            const float mn = fmaxf(m, mx);
            const float corr = m > -INFINITY ? expf(m - mn) : 0.f;        // rows are heads, on both operands
            l *= corr;
#pragma unroll
            for (int i = 0; i < VC; ++i) { o[i][0] *= corr; o[i][1] *= corr; }
            m = mn;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            z[j] = ex2((z[j] - m) * 1.4426950408889634f) * cnt[j];
            l += z[j];
            if (MASS && c.r < p.rep && cnt[j] > 0.f) {   // the block's whole mass is reported as its first unit
                constexpr int UPB = kP / G;
                float2* mp = p.mass_part + ((size_t)it.row * p.nb + orig[j]) * UPB * p.rep + c.r;
                mp[0] = make_float2(m, z[j]);
                for (int u = 1; u < UPB; ++u) mp[(size_t)u * p.rep] = make_float2(-INFINITY, 0.f);
            }
        }
        uint32_t ph[2], pl[2];
        split_f16x2(z[0] * kScale, z[1] * kScale, ph[0], pl[0]);
        split_f16x2(z[2] * kScale, z[3] * kScale, ph[1], pl[1]);
#pragma unroll
        for (int h = 0; h < NV; ++h) {
            const uint32_t x0[4] = {vw[0][h].x, vw[0][h].y, vw[0][h].z, vw[0][h].w}, x1[4] = {vw[1][h].x, vw[1][h].y, vw[1][h].z, vw[1][h].w};
            const uint32_t x2[4] = {vw[2][h].x, vw[2][h].y, vw[2][h].z, vw[2][h].w}, x3[4] = {vw[3][h].x, vw[3][h].y, vw[3][h].z, vw[3][h].w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;
                float d[4];
                mma_f16_z(d, ph[0], pl[0], ph[1], pl[1], prmt(x0[i >> 1], x1[i >> 1], sel), prmt(x2[i >> 1], x3[i >> 1], sel));
                o[8 * h + i][0] += d[0] + d[2];
                o[8 * h + i][1] += d[1] + d[3];
            }
        }
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    if (c.r < p.rep) {
        if (c.t == 0) p.part_ml[rec0 + c.r] = make_float2(m, l);
        if (first < tiles) {                              // the merge does not read the rows of a record without blocks
            float* out = p.part + (rec0 + c.r) * D + 2 * VC * c.t;
#pragma unroll
            for (int i = 0; i < VC; i += 4) {
                float a[4], b[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) { a[k] = o[i + k][0] / kScale; b[k] = o[i + k][1] / kScale; }
                store_run<4>(out + i, a);
                store_run<4>(out + VC + i, b);
            }
        }
    }
}

template <int D, int G, bool DUP, bool MASS>
__device__ void consumer_loop(const Params& p, Smem<D, G>& sm, int* abort_flag) {
    using C = Cfg<D, G>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    Ctx<D, G> c;
    c.r = lane >> 2; c.t = lane & 3; c.lane = lane; c.f = 0.f;
    c.part = DUP && (c.r & 1);
    // Pair pr of the CTA belongs to stream pr & 1; its warps share that stream's blocks with the other two pairs' (ring_item).
    const int pr = warp >> 1, half = warp & 1;
    const int stream = pr & 1;
    int beg = 0;                                    // where the item's blocks begin in the stream
    int code = 0;                                   // non-zero: a wait gave up
    for (int iseq = 0; code == 0; ++iseq) {
        const int is = iseq % kItemSlots, ib = iseq & 1;
        if (!mbar_wait(&sm.item_full[is], (uint32_t)(iseq / kItemSlots) & 1u)) { code = 2; break; }
        const ItemDesc it = sm.item[is];
        if (it.exit) return;
        if (!mbar_wait(&sm.qready[ib], (uint32_t)(iseq >> 1) & 1u)) { code = 3; break; }
        c.qprep = smem_u32(sm.qprep) + (uint32_t)(ib * C::QPREP_BYTES) + (uint32_t)lane * 16u;
        c.f = sm.sf[ib * 16 + (DUP ? c.t : c.r)];
        const size_t rec_idx = (size_t)it.row * p.items_per_row + (size_t)(it.item / p.rows);
        const size_t rec0 = (rec_idx * kConsumerWarps + warp) * p.rep;
        if (it.level == 1) {
            // a short item is the work of a few warps: they take turns
            centroid_item<D, G, MASS>(p, c, it, sm.item_tab + is * kMaxItemBlocks, (warp + 4 * iseq) % kConsumerWarps, sm.sf[ib * 16 + 8 + c.r], rec0);
        }
        else {
            const int end = stream ? it.end_seq1 : it.end_seq0;
            if (it.level == 16) code = ring_item<D, G, 16, DUP, MASS>(p, sm, c, it, stream, pr >> 1, half, beg, end, rec0);
            else if (it.level == 8) code = ring_item<D, G, 8, DUP, MASS>(p, sm, c, it, stream, pr >> 1, half, beg, end, rec0);
            else if (it.level == 4) code = ring_item<D, G, 4, DUP, MASS>(p, sm, c, it, stream, pr >> 1, half, beg, end, rec0);
            else code = ring_item<D, G, 2, DUP, MASS>(p, sm, c, it, stream, pr >> 1, half, beg, end, rec0);
            beg = end;
        }
        if (code) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.item_empty[is]);
        if (*reinterpret_cast<volatile int*>(abort_flag)) return;
    }
    if (code && lane == 0) {
        atomicExch(p.status, code);
        atomicExch(abort_flag, 1);
    }
}

// MASS: the variant that also reports the blocks' softmax mass.  It is a separate instantiation because the few
// extra live values of the reporting measurably slow the plain kernel down (5 % on the 16k-token mix).
template <int D, int G, bool DUP, bool MASS>
__global__ void __launch_bounds__(kThreads, kCtasPerSM) decode_mma_kernel(const __grid_constant__ Params p,
                                                                         const __grid_constant__ TensorMaps tm) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ int abort_flag;
    Smem<D, G> sm(smem_raw);
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kStreams * kNSlot; ++s) {
            mbar_init(&sm.full[s], p.paged || tm.planes_tiled ? 1 : 1 + 32);         // the publishing lane's arrival (+ the copies' bytes) and, where lanes fetch planes, 32 of theirs
            mbar_init(&sm.empty[s], 2);             // the two warps of a pair
        }
        for (int s = 0; s < kItemSlots; ++s) {
            mbar_init(&sm.item_full[s], 1);
            mbar_init(&sm.item_empty[s], kConsumerWarps + kStreams);
        }
        mbar_init(&sm.qready[0], 1);
        mbar_init(&sm.qready[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x < kConsumers) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
    if (threadIdx.x < kConsumers) consumer_loop<D, G, DUP, MASS>(p, sm, &abort_flag);
    // Warp w issues from scheduler w mod 4.  The consumers of stream 0 (pairs 0, 2, 4) sit on schedulers
    // 0 and 1, those of stream 1 on 2 and 3; each producer is put on a scheduler of its OWN stream, so
    // that it gets the issue slots exactly when its consumers are waiting for it.
    else if (threadIdx.x < kConsumers + 32) producer_loop<D, G>(p, tm, sm, 0, &abort_flag);        // warp 12: scheduler 0
    else if (threadIdx.x < kConsumers + 64) query_loop<D, G, DUP>(p, sm, &abort_flag);         // warp 13: scheduler 1
    else if (threadIdx.x < kConsumers + 96) producer_loop<D, G>(p, tm, sm, 1, &abort_flag);        // warp 14: scheduler 2
    else scheduler_loop<D, G>(p, sm, &abort_flag);                                             // warp 15: scheduler 3
}

}  // namespace mma
}  // namespace gkv
