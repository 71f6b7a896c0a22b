// Rate-distortion rung allocator and its distortion table, one CTA per cache row.
//
// The reference (geodesia_kv/policies.py:810-868) sorts all 4*nb marginal-cost ratios and
// bisects over the sorted array for the first candidate threshold whose allocation fits the
// bit budget.  The feasible thresholds form an up-set of the candidate values, so the same
// threshold is found without a sort by bisecting over the order-preserving integer image of
// fp32: the smallest feasible key inside [min candidate, max candidate] is that candidate,
// the min candidate when every threshold fits, the max candidate when none does.  The
// allocation at a threshold takes, per block, the longest prefix (from ladder step 0) of
// available steps whose ratio is <= threshold, so a block that has already left rung 16
// never moves again — the reference's behaviour, kept on purpose.
#include "gkv_common.cuh"
#include "requantise.cuh"

namespace gkv {

constexpr int kAllocThreads = 512;

__device__ __forceinline__ uint32_t float_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct AllocParams {
    const float* mass; const float* E; const int32_t* idx; const uint8_t* hot;
    const double* target_bits; float* ratio; int32_t* tgt;
    float bits[5];
    float mass_power;
    int nb;
    const int32_t* nb_of;      // optional: blocks in use per problem (rows of a ragged batch); the rest keep their rung
    // Table form (block tables of the paged pool): the ladder index, what must stay exact, the blocks in use and
    // the budget follow from the row's rungs and its length, so idx, hot, nb_of and target_bits are not needed.
    const int32_t* level; const int32_t* lens;
    int64_t mass_stride, level_stride;
    int sink_blocks, window_blocks;
    double target_per_block;
};

// What the allocator has to know about block b of a problem.
struct BlockState { int idx; bool hot; };
template <bool TABLE>
__device__ __forceinline__ BlockState block_state(const AllocParams& p, int prob, int b, int len) {
    if (TABLE) {
        const int lv = p.level[(size_t)prob * p.level_stride + b];
        const int nbr = (len + kP - 1) / kP, open = len > 0 ? (len - 1) / kP : -1;
        // sinks, the block being written and its predecessor, the recent window (policies.py:677-681)
        const bool hot = (b < p.sink_blocks || b >= open - 1 || b >= nbr - p.window_blocks) && b < nbr;
        return {(lv <= 8) + (lv <= 4) + (lv <= 2) + (lv <= 1), hot};
    }
    return {p.idx[(size_t)prob * p.nb + b], p.hot[(size_t)prob * p.nb + b] != 0};
}

// Marginal cost of every ladder step of a block: added damage per saved bit, `big` where the step is not open.
__device__ __forceinline__ void step_ratios(const AllocParams& p, float mass, const float* __restrict__ E, const BlockState& st, float (&r)[4]) {
    const float big = 3.4028234663852886e38f / 4.0f;
    float mc = fmaxf(mass, 1e-12f);
    if (p.mass_power != 1.0f) mc = powf(mc, p.mass_power);
    float dmg[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) dmg[c] = __fmul_rn(mc, E[c]);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const float gain = fmaxf(__fsub_rn(p.bits[s], p.bits[s + 1]), 1e-9f);
        const float cost = __fsub_rn(dmg[s + 1], dmg[s]);
        r[s] = ((s >= st.idx) && !st.hot) ? __fdiv_rn(cost, gain) : big;
    }
}

// Ladder index a block lands on at threshold lam: the prefix rule starts at step 0, so a block that has left rung
// 16 (or must stay) does not move.
__device__ __forceinline__ int landing(const float (&r)[4], const BlockState& st, float lam) {
    if (st.idx != 0 || st.hot) return min(st.idx, 4);
    int pref = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
        if (pref == s && r[s] <= lam) pref = s + 1;
    return pref;
}

// The interval of keys [lo, hi] after N thresholds m (ascending) were tried: the first that fits and the last that
// does not close it.
template <int N>
__device__ __forceinline__ void split_points(uint32_t lo, uint32_t hi, uint32_t (&m)[N]) {
#pragma unroll
    for (int c = 0; c < N; ++c) m[c] = lo + (uint32_t)(((unsigned long long)(hi - lo) * (unsigned)(c + 1)) / (unsigned)(N + 1));
}
template <int N>
__device__ __forceinline__ void narrow(const uint32_t (&m)[N], const bool (&ok)[N], uint32_t& lo, uint32_t& hi) {
#pragma unroll
    for (int c = N - 1; c >= 0; --c)
        if (ok[c]) hi = m[c];
#pragma unroll
    for (int c = 0; c < N; ++c)
        if (!ok[c]) lo = m[c] + 1;
}
__device__ __forceinline__ const float* mass_row(const AllocParams& p, int prob, bool table) {
    return p.mass + (size_t)prob * (table ? p.mass_stride : (int64_t)p.nb);
}
template <bool TABLE>
__device__ __forceinline__ float target_of(const AllocParams& p, int prob, int nb_row) {      // fp32 comparison, as torch does
    return TABLE ? (float)((double)nb_row * p.target_per_block) : (float)p.target_bits[prob];
}

// Rows of at most 512 blocks (32k tokens) whose rungs cost whole numbers of bits (every ladder does): one block per
// thread.  Bound: the length of one warp's instruction stream (a row is one CTA with no more warps than it has blocks,
// and nothing else runs on its SM), so a candidate has to be cheap: a block's four ratios become ascending keys once
// (the prefix rule: step s is taken below its own threshold and those before it), a candidate is four compares whose
// votes are counted, and the bits follow from the counts.  64 rows of 128 blocks: 25 -> 8.6 us against seven candidates
// per round with selected bits and a reduction each, 20 us with one candidate in doubles.
template <bool TABLE>
__global__ void __launch_bounds__(kAllocThreads) allocate_small_kernel(const __grid_constant__ AllocParams p) {
    constexpr int kCand = 3;
    __shared__ int sums[2][kCand][kAllocThreads / 32];
    __shared__ uint32_t su[2][kAllocThreads / 32];
    __shared__ int s0[kAllocThreads / 32];
    const int prob = blockIdx.x, b = threadIdx.x, lane = b & 31, warp = b >> 5, nwarp = blockDim.x >> 5;
    const int nb_all = p.nb, len = TABLE ? p.lens[prob] : 0;
    const int nb_row = TABLE ? (len + kP - 1) / kP : p.nb_of ? p.nb_of[prob] : nb_all;
    const int nb = max(0, min(nb_all, nb_row));
    int32_t* tgt = p.tgt + (size_t)prob * nb_all;
    BlockState my{4, true};
    uint32_t kmin = 0xffffffffu, kmax = 0u, key[4] = {~0u, ~0u, ~0u, ~0u};
    const int bits[5] = {(int)p.bits[0], (int)p.bits[1], (int)p.bits[2], (int)p.bits[3], (int)p.bits[4]};
    int mine = 0;                               // bits of this thread's block where it stands
    if (b < nb_all) my = block_state<TABLE>(p, prob, b, len);
    if (b < nb) {
        float r[4];
        step_ratios(p, mass_row(p, prob, TABLE)[b], p.E + ((size_t)prob * nb_all + b) * 5, my, r);
        float* ratio = p.ratio ? p.ratio + ((size_t)prob * nb_all + b) * 4 : nullptr;
        uint32_t top = 0u;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (ratio) ratio[s] = r[s];
            const uint32_t k = float_key(r[s]);
            kmin = min(kmin, k);
            kmax = max(kmax, k);
            // -0 and +0 are the same threshold; a ratio that is not a number is below none
            top = max(top, r[s] == r[s] ? float_key(r[s] + 0.f) : ~0u);
            key[s] = (my.idx == 0 && !my.hot) ? top : ~0u;
        }
        const int id = min(my.idx, 4);
        mine = id == 0 ? bits[0] : id == 1 ? bits[1] : id == 2 ? bits[2] : id == 3 ? bits[3] : bits[4];
    } else if (b < nb_all) {
        tgt[b] = my.idx;
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (nwarp > 1) {
        if (lane == 0) { su[0][warp] = kmin; su[1][warp] = kmax; s0[warp] = mine; }
        __syncthreads();
        kmin = __reduce_min_sync(0xffffffffu, lane < nwarp ? su[0][lane] : ~0u);
        kmax = __reduce_max_sync(0xffffffffu, lane < nwarp ? su[1][lane] : 0u);
        mine = __reduce_add_sync(0xffffffffu, lane < nwarp ? s0[lane] : 0);
    }
    if (nb == 0) return;

    const float target = target_of<TABLE>(p, prob, nb_row);
    const int gain[4] = {bits[0] - bits[1], bits[1] - bits[2], bits[2] - bits[3], bits[3] - bits[4]};
    int par = 0;
    auto fits = [&](const uint32_t (&m)[kCand], bool (&ok)[kCand]) {
        int tot[kCand];
#pragma unroll
        for (int c = 0; c < kCand; ++c) {
            // a threshold that is not a number takes no step (it compares with nothing)
            const uint32_t at = key_float(m[c]) == key_float(m[c]) ? (m[c] == 0x7fffffffu ? 0x80000000u : m[c]) : 0u;
            tot[c] = 0;
#pragma unroll
            for (int s = 0; s < 4; ++s) tot[c] += __popc(__ballot_sync(0xffffffffu, key[s] <= at && key[s] != ~0u)) * gain[s];
        }
        if (nwarp > 1) {
            if (lane == 0)
#pragma unroll
                for (int c = 0; c < kCand; ++c) sums[par][c][warp] = tot[c];
            __syncthreads();                    // two buffers in turn: one barrier per round is enough
#pragma unroll
            for (int c = 0; c < kCand; ++c) tot[c] = __reduce_add_sync(0xffffffffu, lane < nwarp ? sums[par][c][lane] : 0);
            par ^= 1;
        }
#pragma unroll
        for (int c = 0; c < kCand; ++c) ok[c] = !((float)(mine - tot[c]) > target);
    };
    uint32_t lo = kmin, hi = kmax, m[kCand] = {kmax, kmax, kmax};
    bool ok[kCand];
    fits(m, ok);
    if (ok[0]) {
        while (lo < hi) {
            split_points(lo, hi, m);
            fits(m, ok);
            narrow(m, ok, lo, hi);
        }
    }
    if (b < nb) {
        const float lam = key_float(hi);
        const uint32_t at = lam == lam ? (hi == 0x7fffffffu ? 0x80000000u : hi) : 0u;
        int l = min(my.idx, 4);
        if (my.idx == 0 && !my.hot) {
            l = 0;
#pragma unroll
            for (int s = 0; s < 4; ++s) l += key[s] <= at && key[s] != ~0u;
        }
        tgt[b] = l;
    }
}

// Longer rows: the ratios go to memory and are read back in every round, several blocks per thread, sums in doubles (in an
// order that does not depend on the data).
template <bool TABLE>
__global__ void __launch_bounds__(kAllocThreads) allocate_kernel(const __grid_constant__ AllocParams p) {
    constexpr int kCand = 3;
    __shared__ double sums[2][kCand][kAllocThreads / 32];
    __shared__ uint32_t su[2][kAllocThreads / 32];
    const int prob = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nwarp = kAllocThreads / 32;
    const int nb_all = p.nb, len = TABLE ? p.lens[prob] : 0;
    const int nb_row = TABLE ? (len + kP - 1) / kP : p.nb_of ? p.nb_of[prob] : nb_all;
    const int nb = max(0, min(nb_all, nb_row));
    const float* mass = mass_row(p, prob, TABLE);
    const float* E = p.E + (size_t)prob * nb_all * 5;
    float* ratio = p.ratio + (size_t)prob * nb_all * 4;
    int32_t* tgt = p.tgt + (size_t)prob * nb_all;
    for (int b = nb + tid; b < nb_all; b += kAllocThreads) tgt[b] = block_state<TABLE>(p, prob, b, len).idx;

    uint32_t kmin = 0xffffffffu, kmax = 0u;
    for (int b = tid; b < nb; b += kAllocThreads) {
        float r[4];
        step_ratios(p, mass[b], E + b * 5, block_state<TABLE>(p, prob, b, len), r);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            ratio[b * 4 + s] = r[s];
            const uint32_t k = float_key(r[s]);
            kmin = min(kmin, k);
            kmax = max(kmax, k);
        }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) { su[0][warp] = kmin; su[1][warp] = kmax; }
    __syncthreads();                           // also: ratio[] written by this CTA is read back below
    for (int w = 0; w < nwarp; ++w) { kmin = min(kmin, su[0][w]); kmax = max(kmax, su[1][w]); }
    if (nb == 0) return;

    const float target = target_of<TABLE>(p, prob, nb_row);
    auto land = [&](int b, float lam) -> int {
        float r[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) r[s] = ratio[b * 4 + s];
        return landing(r, block_state<TABLE>(p, prob, b, len), lam);
    };
    int par = 0;
    auto fits = [&](const uint32_t (&m)[kCand], bool (&ok)[kCand]) {
        double tot[kCand] = {0.0, 0.0, 0.0};
        for (int b = tid; b < nb; b += kAllocThreads)
#pragma unroll
            for (int c = 0; c < kCand; ++c) {
                const int l = land(b, key_float(m[c]));
                tot[c] += (double)(l == 0 ? p.bits[0] : l == 1 ? p.bits[1] : l == 2 ? p.bits[2] : l == 3 ? p.bits[3] : p.bits[4]);
            }
#pragma unroll
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (int c = 0; c < kCand; ++c) tot[c] += __shfl_xor_sync(0xffffffffu, tot[c], o);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < kCand; ++c) sums[par][c][warp] = tot[c];
        __syncthreads();                       // two buffers in turn: one barrier per round is enough
#pragma unroll
        for (int c = 0; c < kCand; ++c) {
            double r = sums[par][c][0];
            for (int w = 1; w < nwarp; ++w) r += sums[par][c][w];
            ok[c] = !((float)r > target);
        }
        par ^= 1;
    };
    uint32_t lo = kmin, hi = kmax, m[kCand] = {kmax, kmax, kmax};
    bool ok[kCand];
    fits(m, ok);
    if (ok[0]) {
        while (lo < hi) {
            split_points(lo, hi, m);
            fits(m, ok);
            narrow(m, ok, lo, hi);
        }
    }
    const float lam = key_float(hi);
    for (int b = tid; b < nb; b += kAllocThreads) tgt[b] = land(b, lam);
}

// Sums in integers are the doubles' sums when every rung costs a whole number of bits and 512 of them fit 31 bits.
static bool whole_bits(const float (&bits)[5]) {
    for (float b : bits)
        if (!(b >= 0.f && b <= 4194303.f && b == (float)(int)b)) return false;
    return true;
}

// Which of the two kernels: one block per thread and ratios in registers, or ratios in memory.
static bool allocates_in_registers(int nb, const float (&bits)[5]) { return nb <= kAllocThreads && whole_bits(bits); }

template <bool TABLE>
static int launch_allocate(const AllocParams& p, int problems, cudaStream_t stream) {
    if (allocates_in_registers(p.nb, p.bits)) {
        const int threads = (p.nb + 31) & ~31;
        allocate_small_kernel<TABLE><<<problems, threads, 0, stream>>>(p);
    } else {
        allocate_kernel<TABLE><<<problems, kAllocThreads, 0, stream>>>(p);
    }
    GKV_LAUNCH_CHECK();
    return GKV_OK;
}

// ---- distortion table (policies.py:774-808) from rung-16 blocks of the packed cache ------
struct DistParams {
    const uint8_t* data; const int64_t* offs; const int32_t* level; float* E;
    int nb, D, group, per_row_meta;
    float value_weight;
    int64_t stride_bh;
    int tab_stride;            // entries between the rows of offs and level (nb, or the width of a wider table)
};

constexpr int kDistThreads = 256;

__global__ void __launch_bounds__(kDistThreads) distortion_kernel(DistParams p) {
    extern __shared__ float smem[];
    const int D = p.D, tid = threadIdx.x;
    const int kg = min(p.group, kP), vg = min(p.group, D);
    const int G = kP / kg, gv = D / vg;
    // tile rows are padded by one float: several passes below walk a row per thread, and rows an
    // exact multiple of 32 floats apart would all sit in one bank
    const int ld = D + 1;
    float* sk = smem;                    // [64][ld]
    float* sv = sk + kP * ld;            // [64][ld]
    float* rk = sv + kP * ld;            // [G][D]   K ranges
    float* rv = rk + G * D;              // [64][gv] V ranges
    float* mean = rv + kP * gv;          // [2][D]
    float* rad = mean + 2 * D;           // [2][64]
    float* ek = rad + 2 * kP;            // [3][G]
    float* ev = ek + 3 * G;              // [3][64]
    const int blk = blockIdx.x, row = blockIdx.y;
    const int mrow = p.per_row_meta ? row : 0;
    const size_t mi = (size_t)mrow * p.tab_stride + blk;
    float* Eo = p.E + ((size_t)row * p.nb + blk) * 5;
    if (p.level[mi] != 16) {
        if (tid < 5) Eo[tid] = 0.f;
        return;
    }
    const uint16_t* kb = reinterpret_cast<const uint16_t*>(p.data + (size_t)row * p.stride_bh + p.offs[mi]);
    const uint16_t* vb = kb + kP * D;
    if ((reinterpret_cast<uintptr_t>(kb) & 15) == 0) {
        const uint4* k8 = reinterpret_cast<const uint4*>(kb);
        const uint4* v8 = reinterpret_cast<const uint4*>(vb);
        for (int e8 = tid; e8 < kP * D / 8; e8 += kDistThreads) {        // D % 8 == 0: a load stays inside a row
            const int t = (8 * e8) / D, d = 8 * e8 - t * D;
            const uint4 a = k8[e8], b = v8[e8];
            const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sk[t * ld + d + 2 * i] = bf16_bits_to_float(aw[i] & 0xffffu);
                sk[t * ld + d + 2 * i + 1] = bf16_bits_to_float(aw[i] >> 16);
                sv[t * ld + d + 2 * i] = bf16_bits_to_float(bw[i] & 0xffffu);
                sv[t * ld + d + 2 * i + 1] = bf16_bits_to_float(bw[i] >> 16);
            }
        }
    } else {
        for (int e = tid; e < kP * D; e += kDistThreads) {
            const int t = e / D, d = e - t * D;
            sk[t * ld + d] = bf16_bits_to_float(kb[e]);
            sv[t * ld + d] = bf16_bits_to_float(vb[e]);
        }
    }
    __syncthreads();
    for (int u = tid; u < G * D; u += kDistThreads) {
        const int tg = u / D, d = u - tg * D;
        float lo = INFINITY, hi = -INFINITY;
        for (int i = 0; i < kg; ++i) { const float x = sk[(tg * kg + i) * ld + d]; lo = fminf(lo, x); hi = fmaxf(hi, x); }
        rk[u] = __fsub_rn(hi, lo);
    }
    for (int u = tid; u < kP * gv; u += kDistThreads) {
        const int t = u / gv, cg = u - t * gv;
        float lo = INFINITY, hi = -INFINITY;
        for (int i = 0; i < vg; ++i) { const float x = sv[t * ld + cg * vg + i]; lo = fminf(lo, x); hi = fmaxf(hi, x); }
        rv[u] = __fsub_rn(hi, lo);
    }
    for (int u = tid; u < 2 * D; u += kDistThreads) {
        const float* src = u < D ? sk + u : sv + (u - D);
        float s = 0.f;
        for (int t = 0; t < kP; ++t) s = __fadd_rn(s, src[t * ld]);
        mean[u] = __fdiv_rn(s, (float)kP);
    }
    __syncthreads();
    for (int u = tid; u < 2 * kP; u += kDistThreads) {
        const int which = u / kP, t = u - which * kP;
        const float* src = (which ? sv : sk) + t * ld;
        const float* mu = mean + which * D;
        float s = 0.f;
        for (int d = 0; d < D; ++d) { const float x = __fsub_rn(src[d], mu[d]); s = __fadd_rn(s, __fmul_rn(x, x)); }
        rad[u] = __fsqrt_rn(s);
    }
    for (int u = tid; u < 3 * G; u += kDistThreads) {
        const int li = u / G, tg = u - li * G;
        const float den = 2.0f * (float)((1 << (8 >> li)) - 1);
        float s = 0.f;
        for (int d = 0; d < D; ++d) { const float x = __fdiv_rn(rk[tg * D + d], den); s = __fadd_rn(s, __fmul_rn(x, x)); }
        ek[u] = __fsqrt_rn(s);
    }
    for (int u = tid; u < 3 * kP; u += kDistThreads) {
        const int li = u / kP, t = u - li * kP;
        const float den = 2.0f * (float)((1 << (8 >> li)) - 1);
        float s = 0.f;
        for (int cg = 0; cg < gv; ++cg) {
            const float x = __fdiv_rn(rv[t * gv + cg], den);
            s = __fadd_rn(s, __fmul_rn(__fmul_rn(x, x), (float)vg));
        }
        ev[u] = __fsqrt_rn(s);
    }
    __syncthreads();
    if (tid < 5) {
        float a = 0.f, b = 0.f;
        if (tid == 4) {
            for (int t = 0; t < kP; ++t) { a = fmaxf(a, rad[t]); b = fmaxf(b, rad[kP + t]); }
        } else if (tid > 0) {
            const int li = tid - 1;
            for (int tg = 0; tg < G; ++tg) a = fmaxf(a, ek[li * G + tg]);
            for (int t = 0; t < kP; ++t) b = fmaxf(b, ev[li * kP + t]);
        }
        Eo[tid] = __fadd_rn(a, __fmul_rn(p.value_weight, b));
    }
}

// Head dims 64 and 128.  Every sum of the table is a serial fp32 chain in the reference's order (the allocator's
// decisions hang on its last bit), so what bounds a block is the length of those chains, and what bounds the
// launch is how many blocks an SM holds: half a block at a time stays in shared memory as the 16-bit rows it came as
// (17 KB at D = 128, 24 KB with the squares and means), three warps work on it, and nine CTAs fit an SM.  Columns first (a thread owns a channel pair: means, and the K
// ranges by packed minimum and maximum, squared for the three rungs right away), then rows (a thread owns a token; rows are
// padded by 16 bytes, so that eight lanes' 16-byte loads meet no bank twice) while the third warp adds up the
// rungs' squares.  Square roots are monotonic and correctly rounded, so the maxima are taken over the sums.
//
// With value_weight = 0 the V half enters the table as 0 * b, which is 0 unless b is infinite or not a number;
// b is finite if all |V| are below 2^40, so V is then only looked over, and worked through only if that fails.
constexpr int kDistRowThreads = 96;
template <int D>
struct DistSmem {
    static constexpr int LDB = 2 * D + 16;         // bytes per token row
    static constexpr int LDQ = D + 4;              // floats per row of squares
    alignas(16) uint8_t tile[kP * LDB];
    alignas(16) float mean[D];
    alignas(16) float sq[3 * 4 * LDQ];             // [rung][token group][channel]
    uint32_t top[8];                               // K: largest sum per rung, of the centroid; V: the same
    int v_large;
};

// Largest of the warp's non-negative sums into *top; one that is not a number counts as nothing, as in fmaxf.
__device__ __forceinline__ void keep_max(uint32_t* top, float sum) {
    const uint32_t u = __reduce_max_sync(0xffffffffu, sum == sum ? __float_as_uint(sum) : 0u);
    if ((threadIdx.x & 31) == 0) atomicMax(top, u);
}

// Half a block on its way into the tile: asynchronous copies, so that they overlap with whatever follows up to
// distortion_half (which waits for them).
template <int D>
__device__ __forceinline__ void distortion_load(const uint8_t* __restrict__ src, DistSmem<D>& sm) {
    constexpr int LDB = DistSmem<D>::LDB, OPR = D / 8;
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        const uint32_t tile = (uint32_t)__cvta_generic_to_shared(sm.tile);
        for (int e = threadIdx.x; e < kP * OPR; e += kDistRowThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tile + (uint32_t)((e / OPR) * LDB + (e % OPR) * 16)), "l"(src + 16 * e) : "memory");
    } else {
        for (int e = threadIdx.x; e < kP * D; e += kDistRowThreads)
            reinterpret_cast<uint16_t*>(sm.tile + (e / D) * LDB)[e % D] = reinterpret_cast<const uint16_t*>(src)[e];
    }
}

template <int D, bool VALUES>
__device__ __forceinline__ void distortion_half(DistSmem<D>& sm, int kg, int vg) {
    constexpr int LDB = DistSmem<D>::LDB, LDQ = DistSmem<D>::LDQ, OPR = D / 8;
    const int tid = threadIdx.x, lane = tid & 31, G = kP / kg;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (tid < D / 2) {
        float s0 = 0.f, s1 = 0.f;
        const uint8_t* col = sm.tile + 4 * tid;
        for (int tg = 0; tg < G; ++tg) {
            uint32_t lo = 0x7F807F80u, hi = 0xFF80FF80u;       // +inf, -inf
            for (int i0 = 0; i0 < kg; i0 += 16) {
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = *reinterpret_cast<const uint32_t*>(col + (tg * kg + i0 + i) * LDB);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    s0 = __fadd_rn(s0, __uint_as_float(w[i] << 16));
                    s1 = __fadd_rn(s1, __uint_as_float(w[i] & 0xffff0000u));
                    if (!VALUES) { lo = rq::min2<1>(lo, w[i]); hi = rq::max2<1>(hi, w[i]); }
                }
            }
            if (!VALUES) {
                const float r0 = __fsub_rn(__uint_as_float(hi << 16), __uint_as_float(lo << 16));
                const float r1 = __fsub_rn(__uint_as_float(hi & 0xffff0000u), __uint_as_float(lo & 0xffff0000u));
#pragma unroll
                for (int li = 0; li < 3; ++li) {
                    const float den = 2.0f * (float)((1 << (8 >> li)) - 1);
                    const float a = __fdiv_rn(r0, den), b = __fdiv_rn(r1, den);
                    *reinterpret_cast<float2*>(sm.sq + (li * G + tg) * LDQ + 2 * tid) = make_float2(__fmul_rn(a, a), __fmul_rn(b, b));
                }
            }
        }
        *reinterpret_cast<float2*>(sm.mean + 2 * tid) = make_float2(__fdiv_rn(s0, (float)kP), __fdiv_rn(s1, (float)kP));
    }
    __syncthreads();
    if (tid < kP) {
        const uint8_t* row = sm.tile + tid * LDB;
        float s = 0.f, e[3] = {0.f, 0.f, 0.f};
        uint32_t lo = 0x7F807F80u, hi = 0xFF80FF80u;
#pragma unroll 2
        for (int o = 0; o < OPR; ++o) {
            const uint4 r = *reinterpret_cast<const uint4*>(row + 16 * o);
            const float4 m0 = *reinterpret_cast<const float4*>(sm.mean + 8 * o), m1 = *reinterpret_cast<const float4*>(sm.mean + 8 * o + 4);
            const uint32_t w[4] = {r.x, r.y, r.z, r.w};
            const float mu[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float x0 = __fsub_rn(__uint_as_float(w[c] << 16), mu[2 * c]);
                const float x1 = __fsub_rn(__uint_as_float(w[c] & 0xffff0000u), mu[2 * c + 1]);
                s = __fadd_rn(s, __fmul_rn(x0, x0));
                s = __fadd_rn(s, __fmul_rn(x1, x1));
                if (VALUES) { lo = rq::min2<1>(lo, w[c]); hi = rq::max2<1>(hi, w[c]); }
            }
            if (VALUES && (8 * o + 8) % vg == 0) {             // the end of a channel group
                const float h = fmaxf(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u));
                const float l = fminf(__uint_as_float(lo << 16), __uint_as_float(lo & 0xffff0000u));
                const float range = __fsub_rn(h, l);
#pragma unroll
                for (int li = 0; li < 3; ++li) {
                    const float x = __fdiv_rn(range, 2.0f * (float)((1 << (8 >> li)) - 1));
                    e[li] = __fadd_rn(e[li], __fmul_rn(__fmul_rn(x, x), (float)vg));
                }
                lo = 0x7F807F80u; hi = 0xFF80FF80u;
            }
        }
        keep_max(&sm.top[VALUES ? 7 : 3], s);
        if (VALUES)
#pragma unroll
            for (int li = 0; li < 3; ++li) keep_max(&sm.top[4 + li], e[li]);
    } else if (!VALUES) {                                      // the third warp: one lane per (rung, token group)
        float s = 0.f;
        if (lane < 3 * G) {
            const float4* q = reinterpret_cast<const float4*>(sm.sq + lane * LDQ);
#pragma unroll 8
            for (int d = 0; d < D / 4; ++d) {
                const float4 v = q[d];
                s = __fadd_rn(s, v.x); s = __fadd_rn(s, v.y); s = __fadd_rn(s, v.z); s = __fadd_rn(s, v.w);
            }
        }
#pragma unroll
        for (int li = 0; li < 3; ++li) keep_max(&sm.top[li], lane / G == li ? s : 0.f);
    }
    __syncthreads();
}

template <int D>
__global__ void __launch_bounds__(kDistRowThreads) distortion_rows_kernel(DistParams p) {
    __shared__ DistSmem<D> sm;
    const int tid = threadIdx.x;
    const int kg = min(p.group, kP), vg = min(p.group, D);
    const int blk = blockIdx.x, row = blockIdx.y;
    const size_t mi = (size_t)(p.per_row_meta ? row : 0) * p.tab_stride + blk;
    float* Eo = p.E + ((size_t)row * p.nb + blk) * 5;
    if (p.level[mi] != 16) {
        if (tid < 5) Eo[tid] = 0.f;
        return;
    }
    const uint8_t* kb = p.data + (size_t)row * p.stride_bh + p.offs[mi];
    const uint8_t* vb = kb + kP * D * 2;
    if (tid < 8) sm.top[tid] = 0u;
    if (tid == 0) sm.v_large = 0;
    bool need_v = p.value_weight != 0.f;
    distortion_load<D>(kb, sm);
    if (!need_v) {
        uint32_t big = 0u;
        if ((reinterpret_cast<uintptr_t>(vb) & 15) == 0) {
#pragma unroll 11
            for (int e = tid; e < kP * D / 8; e += kDistRowThreads) {
                const uint4 r = reinterpret_cast<const uint4*>(vb)[e];
                big = __vmaxu2(__vmaxu2(__vmaxu2(big, r.x & 0x7fff7fffu), __vmaxu2(r.y & 0x7fff7fffu, r.z & 0x7fff7fffu)), r.w & 0x7fff7fffu);
            }
        } else {
            for (int e = tid; e < kP * D; e += kDistRowThreads) big = max(big, (uint32_t)reinterpret_cast<const uint16_t*>(vb)[e] & 0x7fffu);
        }
        __syncthreads();
        constexpr uint32_t k2p40 = (127u + 40u) << 7;          // 2^40 as bf16
        if ((big & 0xffffu) >= k2p40 || (big >> 16) >= k2p40) sm.v_large = 1;
    }
    distortion_half<D, false>(sm, kg, vg);                     // its barriers also publish v_large
    need_v = need_v || sm.v_large != 0;
    if (need_v) {
        distortion_load<D>(vb, sm);
        distortion_half<D, true>(sm, kg, vg);
    }
    if (tid < 5) {
        float a = 0.f, b = 0.f;
        if (tid > 0) {
            a = __fsqrt_rn(__uint_as_float(sm.top[tid - 1]));
            b = need_v ? __fsqrt_rn(__uint_as_float(sm.top[3 + tid])) : 0.f;
        }
        Eo[tid] = __fadd_rn(a, __fmul_rn(p.value_weight, b));
    }
}

static int launch_distortion(const DistParams& p, int rows, cudaStream_t stream) {
    const int nb = p.nb, D = p.D;
    const int kg = min(p.group, kP), vg = min(p.group, D);
    const int G = kP / kg, gv = D / vg;
    if (rq::shape_ok(D, p.group)) {
        if (p.D == 128) distortion_rows_kernel<128><<<dim3(nb, rows), kDistRowThreads, 0, stream>>>(p);
        else distortion_rows_kernel<64><<<dim3(nb, rows), kDistRowThreads, 0, stream>>>(p);
        GKV_LAUNCH_CHECK();
        return GKV_OK;
    }
    const size_t smem = sizeof(float) * ((size_t)2 * kP * (D + 1) + (size_t)G * D + (size_t)kP * gv + 2 * D + 2 * kP + 3 * G + 3 * kP);
    const size_t smem_max = sizeof(float) * ((size_t)2 * kP * (kMaxD + 1) + (size_t)kP * kMaxD + (size_t)kP * kMaxD + 2 * kMaxD + 2 * kP + 3 * kP + 3 * kP);
    GKV_CUDA_TRY(cudaFuncSetAttribute(distortion_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(smem_max > 227 * 1024 ? 227 * 1024 : smem_max)));
    if (smem > 227 * 1024) return GKV_E_SHAPE;
    distortion_kernel<<<dim3(nb, rows), kDistThreads, smem, stream>>>(p);
    GKV_LAUNCH_CHECK();
    return GKV_OK;
}

}  // namespace gkv

extern "C" {

int gkv_allocate(const float* mass, const float* E, const int32_t* idx, const uint8_t* hot,
                 const float* bits_host, const double* target_bits, float mass_power, float* ratio,
                 int32_t* tgt_idx, int problems, int nb, void* stream) {
    return gkv_allocate_ragged(mass, E, idx, hot, bits_host, target_bits, mass_power, ratio, tgt_idx, nullptr,
                               problems, nb, stream);
}

int gkv_allocate_ragged(const float* mass, const float* E, const int32_t* idx, const uint8_t* hot,
                        const float* bits_host, const double* target_bits, float mass_power, float* ratio,
                        int32_t* tgt_idx, const int32_t* nb_of, int problems, int nb, void* stream) {
    using namespace gkv;
    if (problems <= 0 || nb < 0) return GKV_E_SHAPE;
    if (!bits_host) return GKV_E_NULL;
    if (nb == 0) return GKV_OK;
    if (!mass || !E || !idx || !hot || !target_bits || !ratio || !tgt_idx) return GKV_E_NULL;
    AllocParams p;
    p.mass = mass; p.E = E; p.idx = idx; p.hot = hot; p.target_bits = target_bits; p.ratio = ratio;
    p.tgt = tgt_idx; p.mass_power = mass_power; p.nb = nb; p.nb_of = nb_of;
    for (int i = 0; i < 5; ++i) p.bits[i] = bits_host[i];
    p.level = nullptr; p.lens = nullptr; p.mass_stride = p.level_stride = nb;
    p.sink_blocks = p.window_blocks = 0; p.target_per_block = 0.0;
    return launch_allocate<false>(p, problems, (cudaStream_t)stream);
}

int gkv_block_distortion(const uint8_t* data, const int64_t* offs, const int32_t* level, float* E, int rows,
                         int nb, int D, int block, int group, float value_weight, int64_t stride_bh,
                         int meta_rows, void* stream) {
    using namespace gkv;
    if (block != kP) return GKV_E_BLOCK;
    if (rows <= 0 || nb <= 0 || D <= 0 || D > kMaxD || D % 8 || group <= 0) return GKV_E_SHAPE;
    if (kP % min(group, kP) || D % min(group, D)) return GKV_E_SHAPE;
    if (meta_rows != 1 && meta_rows != rows) return GKV_E_SHAPE;
    if (!data || !offs || !level || !E) return GKV_E_NULL;
    DistParams p;
    p.data = data; p.offs = offs; p.level = level; p.E = E; p.nb = nb; p.D = D; p.group = group;
    p.per_row_meta = meta_rows != 1; p.value_weight = value_weight; p.stride_bh = stride_bh; p.tab_stride = nb;
    return launch_distortion(p, rows, (cudaStream_t)stream);
}

size_t gkv_paged_plan_ratio_bytes(const float* bits_host, int rows, int nb) {
    if (!bits_host || rows <= 0 || nb <= 0) return 0;
    float bits[5];
    for (int i = 0; i < 5; ++i) bits[i] = bits_host[i];
    return gkv::allocates_in_registers(nb, bits) ? 0 : (size_t)rows * nb * 4 * sizeof(float);
}

int gkv_paged_plan_demotion(const uint8_t* pool, const int64_t* offs, const int32_t* level, const int32_t* lens,
                            const float* mass, int64_t mass_stride, const float* bits_host, double target_per_block,
                            int sink_blocks, int window_blocks, float mass_power, float value_weight, float* E,
                            float* ratio, int32_t* tgt_idx, int rows, int nb, int cap, int D, int block, int group,
                            void* stream) {
    using namespace gkv;
    if (block != kP) return GKV_E_BLOCK;
    if (rows <= 0 || nb < 0 || cap < nb || !rq::shape_ok(D, group)) return GKV_E_SHAPE;
    if (nb == 0) return GKV_OK;
    if (mass_stride < nb) return GKV_E_ARG;
    if (!pool || !offs || !level || !lens || !mass || !bits_host || !E || !tgt_idx) return GKV_E_NULL;
    const bool in_registers = gkv_paged_plan_ratio_bytes(bits_host, rows, nb) == 0;
    if (!in_registers && !ratio) return GKV_E_NULL;
    DistParams d;
    d.data = pool; d.offs = offs; d.level = level; d.E = E; d.nb = nb; d.D = D; d.group = group;
    d.per_row_meta = 1; d.value_weight = value_weight; d.stride_bh = 0; d.tab_stride = cap;
    if (const int rc = launch_distortion(d, rows, (cudaStream_t)stream)) return rc;
    AllocParams p;
    p.mass = mass; p.E = E; p.idx = nullptr; p.hot = nullptr; p.target_bits = nullptr;
    p.ratio = in_registers ? nullptr : ratio; p.tgt = tgt_idx; p.mass_power = mass_power; p.nb = nb; p.nb_of = nullptr;
    for (int i = 0; i < 5; ++i) p.bits[i] = bits_host[i];
    p.level = level; p.lens = lens; p.mass_stride = mass_stride; p.level_stride = cap;
    p.sink_blocks = sink_blocks; p.window_blocks = window_blocks; p.target_per_block = target_per_block;
    return launch_allocate<true>(p, rows, (cudaStream_t)stream);
}

}  // extern "C"
