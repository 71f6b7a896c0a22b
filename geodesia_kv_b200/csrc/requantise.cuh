// (Re)quantisation of one 64-token block: the work of the pack and demote kernels for head dims 64 and 128.
//
// A CTA of 256 threads takes one block.  Two bodies:
//   * `requantise`, for fp32 rows: thread (tr, c8) holds eight consecutive channels (8*c8 .. 8*c8+7) of the tokens tr,
//     tr + ROWS, ... of K and of V in registers, so all of a block's global loads are in flight at once and no fp32 tile is
//     staged in shared memory.  K ranges (per channel over `group` consecutive tokens) are reduced in the thread, across the
//     lanes that hold the same channels, and across warps with integer min/max atomics on the order-preserving image of fp32
//     in shared memory; V ranges (per token over `group` consecutive channels) live inside a few neighbouring lanes.
//   * `requantise_staged`, for 16-bit rows and packed blocks, which a bulk copy has put into shared memory: passes read the
//     source again instead of holding it, K ranges leave a warp as partial rows, V is worked out a quarter row per thread.
// In both, codes come out eight per thread and token, as one 8/4/2-byte store in exactly the block's byte order.
//
// The arithmetic is the reference's (geodesia_kv/policies.py:61-77 quant_grouped, packed.py:14-44):
// step = max(hi - lo, 1e-8) / qmax in fp32, lo and step rounded to fp16, code = clamp(rint((x - lo16)
// / step16), 0, qmax) with the quotient rounded as an IEEE division rounds it, centroid = fp32 sum of
// the 64 tokens in order, divided once, rounded to fp16.
#pragma once

#include "gkv_common.cuh"

namespace gkv {
namespace rq {

constexpr int kThreads = 256;

struct Job {
    // source of `requantise`: dense fp32 rows (`requantise_staged` is told its source by a StagedSrc)
    const void* ksrc;           // first token row of the block
    const void* vsrc;
    int64_t src_stride;         // elements between consecutive tokens
    int nvalid;                 // rows beyond nvalid repeat row nvalid - 1
    // destination
    uint8_t* dst;
    int level;
    __half* klo; __half* kstep; __half* vlo; __half* vstep;     // written for rungs 8/4/2; zeroed for 16/1 when zero_scales
    int zero_scales;
    float* ek; float* ev;       // optional: += max over tokens of |x_t - q(x_t)|_2 for K and for V (policies.py:905-906)
    int group;
};

struct __align__(16) Shared {
    uint32_t kmin[4 * 128];     // [G][D] order-preserving keys
    uint32_t kmax[4 * 128];
    float4 ks[4 * 128];         // [G][D] (lo16, step16, 1 / step16) as fp32
    uint32_t err[2];            // max error norms (bits of non-negative floats)
    float csum[2][kP];          // centroid target: per-token squared error sums
};

__device__ __forceinline__ uint32_t fkey(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float keyf(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// code = clamp(rint((x - lo) / step), 0, qmax), the quotient as IEEE division rounds it: the product
// with a reciprocal is within a few ulp of it (absolute error < 1e-4 for quotients up to 255), so it
// rounds to the same integer unless it lands within 1e-3 of a tie, and only then — or when it is huge
// or not a number — is the exact division needed.
__device__ __forceinline__ uint32_t code_of(float x, float lf, float sf, float rs, float qmax) {
    // rounding to nearest-even by adding 1.5 * 2^23 (the integer then sits in the low mantissa bits) keeps
    // the work on the full-rate pipes; valid for |q| < 2^22
    constexpr float kMagic = 12582912.0f;
    const float a = __fsub_rn(x, lf);
    float q = __fmul_rn(a, rs);
    float m = __fadd_rn(q, kMagic);
    float c = __fsub_rn(m, kMagic);
    if (!(fabsf(q - c) < 0.499f) || !(fabsf(q) < 1e6f)) {
        q = __fdiv_rn(a, sf);
        c = rintf(q);
        c = (c != c) ? 0.f : fminf(fmaxf(c, 0.f), qmax);
        return (uint32_t)c;
    }
    const int ci = __float_as_int(m) - 0x4B400000;
    return (uint32_t)min(max(ci, 0), (int)qmax);
}

__device__ __forceinline__ void unpack8_16(const uint4 r, bool bf, float* out) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
    if (bf) {                                   // one branch for the eight values, not one per pair
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            out[2 * i] = __uint_as_float(w[i] << 16);
            out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            out[2 * i] = f.x;
            out[2 * i + 1] = f.y;
        }
    }
}

// Eight channels (8*c8 ..) of token t of the K (which = 0) or V (which = 1) rows, fp32.
__device__ __forceinline__ void load8(const Job& j, int which, int t, int c8, float* out) {
    const float* x = static_cast<const float*>(which ? j.vsrc : j.ksrc) + (size_t)min(t, j.nvalid - 1) * (size_t)j.src_stride + 8 * c8;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const float4 a = reinterpret_cast<const float4*>(x)[0], b = reinterpret_cast<const float4*>(x)[1];
        out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
        out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = x[i];
    }
}

// One element (token t, channel d) of the rows — the centroid path walks a channel token by token.
__device__ __forceinline__ float load1(const Job& j, int which, int t, int d) {
    return static_cast<const float*>(which ? j.vsrc : j.ksrc)[(size_t)min(t, j.nvalid - 1) * (size_t)j.src_stride + d];
}

// Eight codes of `lv` bits each -> lv bytes at `out` (byte order of the block).
__device__ __forceinline__ void store_codes(uint8_t* out, const uint32_t* c, int lv) {
    if (lv == 8) {
        const uint32_t a = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
        const uint32_t b = c[4] | (c[5] << 8) | (c[6] << 16) | (c[7] << 24);
        if ((reinterpret_cast<uintptr_t>(out) & 7) == 0) *reinterpret_cast<uint2*>(out) = make_uint2(a, b);
        else for (int i = 0; i < 8; ++i) out[i] = (uint8_t)c[i];
    } else if (lv == 4) {
        uint32_t w = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) w |= c[i] << (4 * i);
        if ((reinterpret_cast<uintptr_t>(out) & 3) == 0) *reinterpret_cast<uint32_t*>(out) = w;
        else for (int i = 0; i < 4; ++i) out[i] = (uint8_t)(w >> (8 * i));
    } else {
        uint32_t w = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) w |= c[i] << (2 * i);
        if ((reinterpret_cast<uintptr_t>(out) & 1) == 0) *reinterpret_cast<uint16_t*>(out) = (uint16_t)w;
        else { out[0] = (uint8_t)w; out[1] = (uint8_t)(w >> 8); }
    }
}

// Shapes this path takes: D 64 or 128, group 16, 32, 64 or a multiple of 8 from D up.
__host__ __device__ __forceinline__ bool shape_ok(int D, int group) {
    if (D != 64 && D != 128) return false;
    const int kg = group < kP ? group : kP, vg = group < D ? group : D;
    return group % 8 == 0 && kP % kg == 0 && D % vg == 0 && kP / kg <= 4;
}

template <int D>
__device__ void requantise(const Job& j, Shared& sm) {
    constexpr int OPR = D / 8;                 // channel octets per token row
    constexpr int ROWS = kThreads / OPR;       // token rows the CTA covers per pass
    constexpr int NI = kP / ROWS;              // passes: tokens tr, tr + ROWS, ...
    const int tid = threadIdx.x, lane = tid & 31;
    const int c8 = tid % OPR, tr = tid / OPR;
    const int lv = j.level;
    const int kg = min(j.group, kP), vg = min(j.group, D);
    const int G = kP / kg, gv = D / vg;
    const bool quant = lv == 8 || lv == 4 || lv == 2;
    const bool radii = j.ek != nullptr;

    if (tid < 2) sm.err[tid] = 0u;
    if (quant) {
        for (int u = tid; u < G * D; u += kThreads) { sm.kmin[u] = 0xffffffffu; sm.kmax[u] = 0u; }
    } else if (j.zero_scales) {
        // the dense side tensors of the reference hold zeros for rungs 16 and 1 (pack_layout.py:25-28)
        for (int u = tid; u < G * D; u += kThreads) { j.klo[u] = __ushort_as_half(0); j.kstep[u] = __ushort_as_half(0); }
        for (int u = tid; u < kP * gv; u += kThreads) { j.vlo[u] = __ushort_as_half(0); j.vstep[u] = __ushort_as_half(0); }
    }

    if (lv == 1) {
        // centroid: thread (which, d) adds the 64 tokens of its channel in order
        float mean = 0.f;
        const int which = tid / D, d = tid - which * D;
        if (tid < 2 * D) {
            float s = 0.f;
#pragma unroll 8
            for (int t = 0; t < kP; ++t) s = __fadd_rn(s, load1(j, which, t, d));
            mean = __half2float(__float2half_rn(__fdiv_rn(s, (float)kP)));
        }
        if (radii) for (int u = tid; u < 2 * kP; u += kThreads) sm.csum[u / kP][u % kP] = 0.f;
        __syncthreads();                       // every source byte has been read (the destination may overlap it)
        if (radii && tid < 2 * D) {
            for (int t = 0; t < kP; ++t) {
                const float e = __fsub_rn(load1(j, which, t, d), mean);
                float s = e * e;
#pragma unroll
                for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) atomicAdd(&sm.csum[which][t], s);
            }
        }
        __syncthreads();
        if (tid < 2 * D) {
            __half* o = reinterpret_cast<__half*>(j.dst + (which ? half_bytes(1, D) : 0));
            o[d] = __float2half_rn(mean);
        }
        if (radii && tid < 2) {
            float m = 0.f;
            for (int t = 0; t < kP; ++t) m = fmaxf(m, sm.csum[tid][t]);
            float* acc = tid ? j.ev : j.ek;
            *acc += sqrtf(m);
        }
        return;
    }

    // ---- all loads first ------------------------------------------------------------------
    float kx[NI][8], vx[NI][8];
#pragma unroll
    for (int i = 0; i < NI; ++i) load8(j, 0, tr + i * ROWS, c8, kx[i]);
#pragma unroll
    for (int i = 0; i < NI; ++i) load8(j, 1, tr + i * ROWS, c8, vx[i]);
    auto values = [&](int which, int i, float* out) {
#pragma unroll
        for (int c = 0; c < 8; ++c) out[c] = which ? vx[i][c] : kx[i][c];
    };

    if (lv == 16) {
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            uint16_t* half = reinterpret_cast<uint16_t*>(j.dst + (w ? half_bytes(16, D) : 0));
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                float x[8];
                values(w, i, x);
                uint32_t o[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(x[2 * c], x[2 * c + 1]);
                    o[c] = *reinterpret_cast<const uint32_t*>(&b);
                }
                uint16_t* p = half + (size_t)(tr + i * ROWS) * D + 8 * c8;
                if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2], o[3]);
                else for (int c = 0; c < 4; ++c) { p[2 * c] = (uint16_t)o[c]; p[2 * c + 1] = (uint16_t)(o[c] >> 16); }
            }
        }
        return;
    }

    const float qmax = (float)((1 << lv) - 1);
    __syncthreads();                           // key tables initialised

    // ---- K ranges: thread, then the lanes with the same channels, then shared-memory atomics -------
    {
        int cur = tr / kg;
        float lo[8], hi[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) { lo[c] = INFINITY; hi[c] = -INFINITY; }
#pragma unroll
        for (int i = 0; i <= NI; ++i) {
            const int tg = i < NI ? (tr + i * ROWS) / kg : -1;
            if (tg != cur) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
#pragma unroll
                    for (int o = OPR; o < 32; o <<= 1) {
                        lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                        hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
                    }
                    if (lane < OPR) {
                        atomicMin(&sm.kmin[cur * D + 8 * c8 + c], fkey(lo[c]));
                        atomicMax(&sm.kmax[cur * D + 8 * c8 + c], fkey(hi[c]));
                    }
                    lo[c] = INFINITY; hi[c] = -INFINITY;
                }
                cur = tg;
            }
            if (i < NI) {
                float x[8];
                values(0, i, x);
#pragma unroll
                for (int c = 0; c < 8; ++c) { lo[c] = fminf(lo[c], x[c]); hi[c] = fmaxf(hi[c], x[c]); }
            }
        }
    }
    __syncthreads();
    for (int u = tid; u < G * D; u += kThreads) {
        const float lo = keyf(sm.kmin[u]), hi = keyf(sm.kmax[u]);
        const float step = __fdiv_rn(fmaxf(__fsub_rn(hi, lo), 1e-8f), qmax);
        const __half l16 = __float2half_rn(lo), s16 = __float2half_rn(step);
        j.klo[u] = l16; j.kstep[u] = s16;
        const float sf = __half2float(s16);
        // a thread later reads the entries of its eight channels: they are laid out so that the 16 (or 8)
        // lanes of a token row read consecutive 16-byte slots
        const int tgu = u / D, du = u - tgu * D;
        sm.ks[(tgu * 8 + (du & 7)) * OPR + (du >> 3)] = make_float4(__half2float(l16), sf, __frcp_rn(sf), 0.f);
    }
    __syncthreads();                           // also: every source byte has been read before the first code is stored

    float ekmax = 0.f, evmax = 0.f;
    // ---- K codes ---------------------------------------------------------------------------
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int t = tr + i * ROWS;
        const float4* sc = sm.ks + (t / kg) * 8 * OPR + c8;
        uint32_t code[8];
        float x[8];
        values(0, i, x);
        float e2 = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float4 ls = sc[c * OPR];
            code[c] = code_of(x[c], ls.x, ls.y, ls.z, qmax);
            if (radii) { const float e = x[c] - __fmaf_rn((float)code[c], ls.y, ls.x); e2 += e * e; }
        }
        store_codes(j.dst + ((size_t)t * D + 8 * c8) * lv / 8, code, lv);
        if (radii) {
#pragma unroll
            for (int o = 1; o < OPR; o <<= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
            ekmax = fmaxf(ekmax, e2);
        }
    }
    // ---- V: ranges inside vg/8 neighbouring lanes, scales, codes ----------------------------------
    uint8_t* vdst = j.dst + half_bytes(lv, D);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int t = tr + i * ROWS;
        float x[8];
        values(1, i, x);
        float lo = INFINITY, hi = -INFINITY;
#pragma unroll
        for (int c = 0; c < 8; ++c) { lo = fminf(lo, x[c]); hi = fmaxf(hi, x[c]); }
        for (int o = 1; o < vg / 8; o <<= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const float step = __fdiv_rn(fmaxf(__fsub_rn(hi, lo), 1e-8f), qmax);
        const __half l16 = __float2half_rn(lo), s16 = __float2half_rn(step);
        const int cg = (8 * c8) / vg;
        if ((8 * c8) % vg == 0) { j.vlo[t * gv + cg] = l16; j.vstep[t * gv + cg] = s16; }
        const float lf = __half2float(l16), sf = __half2float(s16), rs = __frcp_rn(sf);
        uint32_t code[8];
        float e2 = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            code[c] = code_of(x[c], lf, sf, rs, qmax);
            if (radii) { const float e = x[c] - __fmaf_rn((float)code[c], sf, lf); e2 += e * e; }
        }
        store_codes(vdst + ((size_t)t * D + 8 * c8) * lv / 8, code, lv);
        if (radii) {
#pragma unroll
            for (int o = 1; o < OPR; o <<= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
            evmax = fmaxf(evmax, e2);
        }
    }
    if (radii) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            ekmax = fmaxf(ekmax, __shfl_xor_sync(0xffffffffu, ekmax, o));
            evmax = fmaxf(evmax, __shfl_xor_sync(0xffffffffu, evmax, o));
        }
        if (lane == 0) { atomicMax(&sm.err[0], __float_as_uint(ekmax)); atomicMax(&sm.err[1], __float_as_uint(evmax)); }
        __syncthreads();
        if (tid < 2) {
            float* acc = tid ? j.ev : j.ek;
            *acc += sqrtf(__uint_as_float(sm.err[tid]));
        }
    }
}

// ---- the same work on a block that already sits in shared memory ---------------------------------------
// Source: two 16-bit tiles [64][D] (dense bf16/fp16 rows, or a rung-16 block), or a packed block of a
// quantised rung with its four scale planes; everything 16-byte aligned.
// The 256 working threads of a CTA meet at named barrier 1: the CTA may hold more threads (a producer
// warp that feeds the stages), which must not be part of these barriers.
__device__ __forceinline__ void work_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// Work area of a CTA beside its stages.  Small on purpose: with two 32 KB stages it decides whether three CTAs fit an SM.
struct __align__(16) Work {
    uint16_t part[2 * 8 * 128];  // [min, max][warp][D]: K ranges of eight tokens (16-bit sources); centroid: the means as floats
    float2 lr[4 * 128];          // [G][D] low end and code factor of the K groups
    __half s[4 * 128];           // [G][D] step of the K groups
    uint32_t err[2];             // max error norms (bits of non-negative floats)
};

struct StagedSrc {
    const uint8_t* k; const uint8_t* v;     // dense tiles (kind 1 bf16, 2 fp16), or the halves of the packed block (kind 3)
    int kind, nvalid, level;                // level: rung of a packed source (8, 4 or 2)
    const __half* klo; const __half* kstep; const __half* vlo; const __half* vstep;
    int kgs, vgs;                           // log2 of the K token group and of the V channel group (both powers of two)
    float* fpart;                           // packed sources: room for [min, max][warp][D] fp32 K ranges (a free part of the stage)
    uint32_t k32, v32;                      // k and v as shared-memory addresses: plain 32-bit arithmetic, LDS instead of generic loads
};
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

template <int D>
__device__ __forceinline__ void staged8(const StagedSrc& s, int which, int t, int c8, float* out) {
    if (s.kind != 3) {
        const uint4 r = *reinterpret_cast<const uint4*>((which ? s.v : s.k) + ((size_t)min(t, s.nvalid - 1) * D + 8 * c8) * 2);
        unpack8_16(r, s.kind == 1, out);
        return;
    }
    const int lv = s.level;
    const uint8_t* cp = (which ? s.v : s.k) + ((size_t)t * D + 8 * c8) * lv / 8;
    unsigned long long bits;
    if (lv == 8) { const uint2 r = *reinterpret_cast<const uint2*>(cp); bits = ((unsigned long long)r.y << 32) | r.x; }
    else if (lv == 4) bits = *reinterpret_cast<const uint32_t*>(cp);
    else bits = *reinterpret_cast<const uint16_t*>(cp);
    const uint32_t mask = (1u << lv) - 1u;
    if (which == 0) {
        const uint4 lo4 = *reinterpret_cast<const uint4*>(s.klo + (t >> s.kgs) * D + 8 * c8);
        const uint4 st4 = *reinterpret_cast<const uint4*>(s.kstep + (t >> s.kgs) * D + 8 * c8);
        float lo[8], st[8];
        unpack8_16(lo4, false, lo);
        unpack8_16(st4, false, st);
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = __fmaf_rn((float)((uint32_t)(bits >> (i * lv)) & mask), st[i], lo[i]);
    } else {
        const int si = t * (D >> s.vgs) + ((8 * c8) >> s.vgs);
        const float st = __half2float(s.vstep[si]), lo = __half2float(s.vlo[si]);
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = __fmaf_rn((float)((uint32_t)(bits >> (i * lv)) & mask), st, lo);
    }
}

template <int D, int SRC>
__device__ __forceinline__ void staged_octet(const StagedSrc& s, int which, int t, int c8, float* out) {
    if constexpr (SRC != 3)
        unpack8_16(lds128((which ? s.v32 : s.k32) + (uint32_t)((min(t, s.nvalid - 1) * D + 8 * c8) * 2)), SRC == 1, out);
    else
        staged8<D>(s, which, t, c8, out);
}

template <int D>
__device__ __forceinline__ float staged1(const StagedSrc& s, int which, int t, int d) {
    if (s.kind != 3) {
        const uint16_t h = reinterpret_cast<const uint16_t*>(which ? s.v : s.k)[(size_t)min(t, s.nvalid - 1) * D + d];
        return s.kind == 1 ? bf16_bits_to_float(h) : half_bits_to_float(h);
    }
    const float c = (float)unpack_code(which ? s.v : s.k, t * D + d, s.level);
    if (which == 0) {
        const int i = (t >> s.kgs) * D + d;
        return __fmaf_rn(c, __half2float(s.kstep[i]), __half2float(s.klo[i]));
    }
    const int i = t * (D >> s.vgs) + (d >> s.vgs);
    return __fmaf_rn(c, __half2float(s.vstep[i]), __half2float(s.vlo[i]));
}

// ---- quantised target rungs ------------------------------------------------------------------------------
// Bound: instruction issue (16384 elements per block; the bytes alone take 6.6 ns of the chip per 4-bit block).
// What an element costs is therefore counted: a 16-bit source is compared in packed pairs (half an instruction
// per element and side), every thread holds ONE token group of K and ONE stretch of a V row, so ranges need few
// shuffles and no atomics and every division serves 32 elements, and a code is a subtraction, a fused
// multiply-add that rounds it, a three-instruction tie test and a little over one instruction of packing.
// Packed minimum / maximum of two bf16 (SRC 1) or fp16 (SRC 2) values; a NaN operand loses, -0 < +0.
template <int SRC>
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) {
    uint32_t d;
    if (SRC == 1) asm("min.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    else asm("min.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
template <int SRC>
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    uint32_t d;
    if (SRC == 1) asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    else asm("max.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
template <int SRC>
__device__ __forceinline__ float widen(uint16_t h) { return SRC == 1 ? bf16_bits_to_float(h) : half_bits_to_float(h); }

struct Scale { float l, s, r; __half l16, s16; };
// lo and step of a range as the reference defines them (fp32, then rounded to fp16), and the factor r the codes
// are taken with: 1 / step to 2^-23, or NaN where a quotient of the range could leave the 16 bits the codes are
// cut from (a step that rounded to 0 or infinity, a low end whose rounding dwarfs the step) — a NaN factor
// sends every code of the group to the exact division.
template <int LV>
__device__ __forceinline__ Scale scale_of(float lo, float hi) {
    constexpr float qmax = (float)((1 << LV) - 1);
    Scale c;
    const float step = __fdiv_rn(fmaxf(__fsub_rn(hi, lo), 1e-8f), qmax);
    c.l16 = __float2half_rn(lo);
    c.s16 = __float2half_rn(step);
    c.l = __half2float(c.l16);
    c.s = __half2float(c.s16);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(c.s));
    const bool small = fabsf((lo - c.l) * r) < 30000.f && fabsf((hi - c.l) * r) < 30000.f;
    c.r = small ? r : __int_as_float(0x7fffffff);
    return c;
}

// Eight codes of LV bits, packed in block order into w[0..].  code = clamp(rint((x - l) / s), 0, qmax) with the
// quotient rounded as IEEE division rounds it: the product with r is within q * 2^-23 of the quotient and the
// division adds q * 2^-24, so both round to the same integer unless the product lands within (qmax + 1) *
// 2.5e-7 of a tie; only then (or for a NaN) is the division made.  Adding 1.5 * 2^23 inside the fused
// multiply-add rounds to nearest-even and leaves the integer in the low 16 bits (two's complement; quotients
// stay below 30000, see scale_of), where pairs are clamped by one instruction.  Returns the octet's squared
// reconstruction error when RADII.
// NS = 8: a scale per channel; 1: one for the octet.  step_of(c): the step of channel c, which only the exact division
// and the radii need.
template <int LV, bool RADII, int NS, class Step>
__device__ __forceinline__ float codes8(const float (&x)[8], const float (&l)[NS], const float (&r)[NS], const Step& step_of, uint32_t (&w)[LV == 8 ? 2 : 1]) {
    constexpr float kMagic = 12582912.0f, qmax = (float)((1 << LV) - 1), tie = 0.5f - (qmax + 1.0f) * 2.5e-7f;
    float m[8];
    bool redo = false;                         // some quotient is near a tie, or not a number
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float a = __fsub_rn(x[c], l[c % NS]);
        m[c] = __fmaf_rn(a, r[c % NS], kMagic);
        redo = redo | !(fabsf(__fmaf_rn(a, r[c % NS], __fsub_rn(kMagic, m[c]))) < tie);
    }
    if (redo) {
        // 16-bit inputs sit on a coarse grid, so near ties are not that rare: six to ten codes in 10,000, which is
        // every fifth to seventh octet of a warp.  Only those codes are divided, one after the other.
        uint32_t todo = 0u;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float a = __fsub_rn(x[c], l[c % NS]);
            if (!(fabsf(__fmaf_rn(a, r[c % NS], __fsub_rn(kMagic, m[c]))) < tie)) todo |= 1u << c;
        }
#pragma unroll 1
        while (todo) {
            const int at = __ffs((int)todo) - 1;
            todo &= todo - 1u;
            float xa = x[0], la = l[0];
#pragma unroll
            for (int c = 1; c < 8; ++c)
                if (at == c) { xa = x[c]; la = l[c % NS]; }
            const float q = rintf(__fdiv_rn(__fsub_rn(xa, la), step_of(at)));
            const float ma = kMagic + ((q != q) ? 0.f : fminf(fmaxf(q, 0.f), qmax));
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (at == c) m[c] = ma;
        }
    }
    constexpr uint32_t QQ = (uint32_t)((1 << LV) - 1) * 0x00010001u;
    uint32_t p[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {              // 8-bit codes: pairs (0,1) (2,3) ..; narrower: (0,4) (1,5) ..
        const int a = LV == 8 ? 2 * c : c, b = LV == 8 ? 2 * c + 1 : c + 4;
        p[c] = __vimin_s16x2_relu(__byte_perm(__float_as_uint(m[a]), __float_as_uint(m[b]), 0x5410), QQ);
    }
    if constexpr (LV == 8) {
        w[0] = __byte_perm(p[0], p[1], 0x6420);
        w[1] = __byte_perm(p[2], p[3], 0x6420);
    } else if constexpr (LV == 4) {
        w[0] = p[0] + p[1] * 16u + p[2] * 256u + p[3] * 4096u;
    } else {
        w[0] = __byte_perm(p[0] + p[1] * 4u + p[2] * 16u + p[3] * 64u, 0u, 0x4420);
    }
    float e2 = 0.f;
    if constexpr (RADII) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float q = fminf(fmaxf(__fsub_rn(m[c], kMagic), 0.f), qmax);
            const float e = x[c] - __fmaf_rn(q, step_of(c), l[c % NS]);
            e2 += e * e;
        }
    }
    return e2;
}

// An octet's codes at their place in the block (`aligned`: the block's start allows one store).
template <int LV>
__device__ __forceinline__ void store_octet(uint8_t* out, const uint32_t (&w)[LV == 8 ? 2 : 1], bool aligned) {
    if (aligned) {
        if constexpr (LV == 8) *reinterpret_cast<uint2*>(out) = make_uint2(w[0], w[1]);
        else if constexpr (LV == 4) *reinterpret_cast<uint32_t*>(out) = w[0];
        else *reinterpret_cast<uint16_t*>(out) = (uint16_t)w[0];
    } else {
#pragma unroll
        for (int i = 0; i < LV; ++i) out[i] = (uint8_t)(w[i / 4] >> (8 * (i % 4)));
    }
}

// SRC 1 / 2: bf16 / fp16 tiles; 3: a packed block of a quantised rung (values in fp32).
//
// K: thread (tr, c8) holds channels 8*c8 .. +7 of NI consecutive tokens, which lie in one token group (16 tokens
// or more); the lanes of a warp hold eight tokens of every channel, so a warp leaves one row of partial ranges
// in shared memory and a group's range is the best of group / 8 rows.
// V: thread (t, quarter) holds a quarter of token t's row — whole channel groups, or an even share of one.  Its
// octets are taken in an order XORed by the lane, which spreads the eight lanes of a 16-byte phase over all banks
// (rows are 128 or 256 bytes apart).
//
// The loops that make codes are not unrolled: several rungs' bodies run side by side on an SM, and unrolled (3000
// instructions each) they are bound by instruction fetch (41 ns per block of the 10/20/40/20/10 % mix).
//
// Measured, 4096 blocks per launch, bf16 in, D = 128, g = 32, ns per block of the whole chip, with one body for all
// that found K ranges by shared-memory atomics and took every quotient apart from the others' -> so: 8-bit 29.6 -> 19.0,
// 4-bit 29.2 -> 16.1, 2-bit 29.1 -> 16.1, centroid 9.2 -> 8.0, the mix 35.6 -> 16.4.
// With three CTAs of 72 registers per SM instead of two of 96: 8-bit 16.8, 4-bit 15.2, 2-bit 15.2, centroid 7.1, mix 15.8
// (three CTAs with one stage each: 19.5, 17.6, 17.6, 8.9, 17.8).
template <int D, int LV, int SRC, bool RADII>
__device__ __forceinline__ void quantise_staged(const StagedSrc& src, const Job& j, Work& sm) {
    constexpr int OPR = D / 8, NI = kP * OPR / kThreads;       // octets per row; tokens of K per thread
    constexpr bool T16 = SRC != 3;
    constexpr uint32_t PINF = SRC == 2 ? 0x7C007C00u : 0x7F807F80u, NINF = SRC == 2 ? 0xFC00FC00u : 0xFF80FF80u;
    constexpr int NW = LV == 8 ? 2 : 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c8 = tid % OPR, t0 = (tid / OPR) * NI;
    const int kgs = src.kgs, vgs = src.vgs;
    const int G = kP >> kgs, gv = D >> vgs;
    const bool aligned = (reinterpret_cast<uintptr_t>(j.dst) & (uintptr_t)(LV - 1)) == 0;     // octets are LV bytes apart

    // ---- K ranges of the warp's eight tokens -----------------------------------------------------------
    if constexpr (T16) {
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) { lo[c] = PINF; hi[c] = NINF; }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const uint4 raw = lds128(src.k32 + (uint32_t)((min(t0 + i, src.nvalid - 1) * D + 8 * c8) * 2));
            const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) { lo[c] = min2<SRC>(lo[c], w[c]); hi[c] = max2<SRC>(hi[c], w[c]); }
        }
#pragma unroll
        for (int o = OPR; o < 32; o <<= 1)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                lo[c] = min2<SRC>(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                hi[c] = max2<SRC>(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            }
        uint16_t* part = sm.part;                                          // [2][8 warps][D]
        if (lane < OPR) *reinterpret_cast<uint4*>(part + warp * D + 8 * c8) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        else if (lane < 2 * OPR) *reinterpret_cast<uint4*>(part + (8 + warp) * D + 8 * c8) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    } else {
        float lo[8], hi[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) { lo[c] = INFINITY; hi[c] = -INFINITY; }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            float x[8];
            staged8<D>(src, 0, t0 + i, c8, x);
#pragma unroll
            for (int c = 0; c < 8; ++c) { lo[c] = fminf(lo[c], x[c]); hi[c] = fmaxf(hi[c], x[c]); }
        }
#pragma unroll
        for (int o = OPR; o < 32; o <<= 1)
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            }
        if (lane < OPR) {
            float4* part = reinterpret_cast<float4*>(src.fpart + warp * D + 8 * c8);
            part[0] = make_float4(lo[0], lo[1], lo[2], lo[3]); part[1] = make_float4(lo[4], lo[5], lo[6], lo[7]);
        } else if (lane < 2 * OPR) {
            float4* part = reinterpret_cast<float4*>(src.fpart + (8 + warp) * D + 8 * c8);
            part[0] = make_float4(hi[0], hi[1], hi[2], hi[3]); part[1] = make_float4(hi[4], hi[5], hi[6], hi[7]);
        }
    }

    float ekmax = 0.f, evmax = 0.f;
    // ---- V: ranges, scales, codes — done here, between the K partials and the barrier that publishes them, so
    // that warps which finish early have work instead of a wait
    {
        constexpr int E = D / 4, NO = E / 8;                   // channels and octets per thread
        constexpr int NSET = NO >= 4 ? 2 : 1;                  // 16-channel stretches that can be groups of their own
        constexpr int ES = E / NSET, OS = NO / NSET;
        const int t = tid >> 2, q4 = tid & 3;
        const int f = NO == 4 ? (lane >> 1) & 3 : (lane >> 2) & 1;
        float lo[NSET], hi[NSET];
#pragma unroll
        for (int st = 0; st < NSET; ++st) {
            if constexpr (T16) {
                uint32_t a = PINF, b = NINF;
                const uint32_t row = src.v32 + (uint32_t)((min(t, src.nvalid - 1) * D + q4 * E) * 2);
#pragma unroll
                for (int o = st * OS; o < (st + 1) * OS; ++o) {
                    const uint4 r = lds128(row + (uint32_t)(16 * (o ^ f)));
                    a = min2<SRC>(min2<SRC>(a, min2<SRC>(r.x, r.y)), min2<SRC>(r.z, r.w));
                    b = max2<SRC>(max2<SRC>(b, max2<SRC>(r.x, r.y)), max2<SRC>(r.z, r.w));
                }
                lo[st] = fminf(fminf(INFINITY, widen<SRC>((uint16_t)a)), widen<SRC>((uint16_t)(a >> 16)));
                hi[st] = fmaxf(fmaxf(-INFINITY, widen<SRC>((uint16_t)b)), widen<SRC>((uint16_t)(b >> 16)));
            } else {
                lo[st] = INFINITY; hi[st] = -INFINITY;
#pragma unroll
                for (int o = st * OS; o < (st + 1) * OS; ++o) {
                    float x[8];
                    staged8<D>(src, 1, t, q4 * NO + (o ^ f), x);
#pragma unroll
                    for (int c = 0; c < 8; ++c) { lo[st] = fminf(lo[st], x[c]); hi[st] = fmaxf(hi[st], x[c]); }
                }
            }
        }
        Scale sc[NSET];
        if ((1 << vgs) < E) {                                  // 16-channel groups: one per stretch (D = 128)
#pragma unroll
            for (int st = 0; st < NSET; ++st) {
                sc[st] = scale_of<LV>(lo[st], hi[st]);
                const int cg = (q4 * E + ES * (NSET == 2 ? st ^ (f >> 1) : 0)) >> vgs;
                j.vlo[t * gv + cg] = sc[st].l16; j.vstep[t * gv + cg] = sc[st].s16;
            }
        } else {
            float a = lo[0], b = hi[0];
#pragma unroll
            for (int st = 1; st < NSET; ++st) { a = fminf(a, lo[st]); b = fmaxf(b, hi[st]); }
            for (int o = 1; o < (1 << vgs) / E; o <<= 1) {     // the group's other lanes
                a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
                b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
            }
            sc[0] = scale_of<LV>(a, b);
#pragma unroll
            for (int st = 1; st < NSET; ++st) sc[st] = sc[0];
            if (((q4 * E) & ((1 << vgs) - 1)) == 0) {
                const int cg = (q4 * E) >> vgs;
                j.vlo[t * gv + cg] = sc[0].l16; j.vstep[t * gv + cg] = sc[0].s16;
            }
        }
        uint8_t* vdst = j.dst + half_bytes(LV, D) + (t * D + q4 * E) * LV / 8;
        float e2 = 0.f, pair = 0.f;                            // radii: ((o0 + o1) + (o2 + o3)), in the order of the row's octets
#pragma unroll 1
        for (int o = 0; o < NO; ++o) {
            float x[8];
            staged_octet<D, SRC>(src, 1, t, q4 * NO + (o ^ f), x);
            const bool second = NSET == 2 && o >= OS;
            const float l[1] = {second ? sc[NSET - 1].l : sc[0].l}, r[1] = {second ? sc[NSET - 1].r : sc[0].r};
            const float step = second ? sc[NSET - 1].s : sc[0].s;
            uint32_t w[NW];
            const float e = codes8<LV, RADII, 1>(x, l, r, [&](int) { return step; }, w);
            store_octet<LV>(vdst + (o ^ f) * LV, w, aligned);
            if constexpr (RADII) {
                pair = (o & 1) ? pair + e : e;
                if (o & 1) e2 = o == 1 ? pair : e2 + pair;
            }
        }
        if constexpr (RADII) {
            e2 += __shfl_xor_sync(0xffffffffu, e2, 1);
            e2 += __shfl_xor_sync(0xffffffffu, e2, 2);
            evmax = fmaxf(evmax, e2);
        }
    }
    work_sync();
    // ---- K scales: one (token group, channel) per thread and round ----------------------------------------
    for (int u = tid; u < G * D; u += kThreads) {
        const int tg = u / D, d = u % D;
        const int w0 = tg << (kgs - 3), w1 = (tg + 1) << (kgs - 3);        // the group's warps
        float lo = INFINITY, hi = -INFINITY;
        for (int w = w0; w < w1; ++w) {
            if constexpr (T16) {
                lo = fminf(lo, widen<SRC>(sm.part[w * D + d]));
                hi = fmaxf(hi, widen<SRC>(sm.part[(8 + w) * D + d]));
            } else {
                lo = fminf(lo, src.fpart[w * D + d]);
                hi = fmaxf(hi, src.fpart[(8 + w) * D + d]);
            }
        }
        const Scale k = scale_of<LV>(lo, hi);
        j.klo[u] = k.l16; j.kstep[u] = k.s16;
        // a thread reads the entries of its eight channels: the lanes of a token row read consecutive slots
        const int at = (tg * 8 + (d & 7)) * OPR + (d >> 3);
        sm.lr[at] = make_float2(k.l, k.r);
        sm.s[at] = k.s16;
    }
    work_sync();                               // also: every source byte has been read before the first K code is stored

    // ---- K codes ---------------------------------------------------------------------------
    {
        const int at = (t0 >> kgs) * 8 * OPR + c8;
        float l[8], r[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) { const float2 k = sm.lr[at + c * OPR]; l[c] = k.x; r[c] = k.y; }
        auto step_of = [&](int c) { return __half2float(sm.s[at + c * OPR]); };
        uint8_t* kdst = j.dst + (t0 * D + 8 * c8) * LV / 8;
#pragma unroll 1
        for (int i = 0; i < NI; ++i) {
            float x[8];
            staged_octet<D, SRC>(src, 0, t0 + i, c8, x);
            uint32_t w[NW];
            float e2 = codes8<LV, RADII, 8>(x, l, r, step_of, w);
            store_octet<LV>(kdst + i * (D * LV / 8), w, aligned);
            if constexpr (RADII) {
#pragma unroll
                for (int o = 1; o < OPR; o <<= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
                ekmax = fmaxf(ekmax, e2);
            }
        }
    }
    if constexpr (RADII) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            ekmax = fmaxf(ekmax, __shfl_xor_sync(0xffffffffu, ekmax, o));
            evmax = fmaxf(evmax, __shfl_xor_sync(0xffffffffu, evmax, o));
        }
        if (lane == 0) { atomicMax(&sm.err[0], __float_as_uint(ekmax)); atomicMax(&sm.err[1], __float_as_uint(evmax)); }
        work_sync();
        if (tid < 2) {
            float* acc = tid ? j.ev : j.ek;
            *acc += sqrtf(__uint_as_float(sm.err[tid]));
        }
    }
}

// Centroid: the mean of the 64 tokens, added in order.  16-bit sources: a thread owns a channel pair, so a token
// costs it one 4-byte load, two widenings and two additions; what bounds it is the chain of 64 additions.  Radii:
// a thread adds up a quarter of a token's row, as in the V half of the quantised rungs.
template <int D, int SRC, bool RADII>
__device__ __forceinline__ void centroid_staged(const StagedSrc& src, const Job& j, Work& sm) {
    constexpr int E = D / 4, NO = E / 8;
    const int tid = threadIdx.x, lane = tid & 31;
    float* mean = reinterpret_cast<float*>(sm.part);       // [2][D], fp16-rounded
    if constexpr (SRC != 3) {
        if (tid < D) {
            const int which = tid / (D / 2), c = 2 * (tid % (D / 2));
            const uint32_t col = (which ? src.v32 : src.k32) + 2u * c;
            float s0 = 0.f, s1 = 0.f;
            if (src.nvalid >= kP) {
#pragma unroll
                for (int t0 = 0; t0 < kP; t0 += 16) {
                    uint32_t w[16];
#pragma unroll
                    for (int t = 0; t < 16; ++t) w[t] = lds32(col + (uint32_t)((t0 + t) * D * 2));
#pragma unroll
                    for (int t = 0; t < 16; ++t) {
                        s0 = __fadd_rn(s0, widen<SRC>((uint16_t)w[t]));
                        s1 = __fadd_rn(s1, widen<SRC>((uint16_t)(w[t] >> 16)));
                    }
                }
            } else {
#pragma unroll 1
                for (int t = 0; t < kP; ++t) {
                    const uint32_t w = lds32(col + (uint32_t)(min(t, src.nvalid - 1) * D * 2));
                    s0 = __fadd_rn(s0, widen<SRC>((uint16_t)w));
                    s1 = __fadd_rn(s1, widen<SRC>((uint16_t)(w >> 16)));
                }
            }
            const __half h0 = __float2half_rn(__fdiv_rn(s0, (float)kP)), h1 = __float2half_rn(__fdiv_rn(s1, (float)kP));
            __half* o = reinterpret_cast<__half*>(j.dst + (which ? half_bytes(1, D) : 0)) + c;
            if ((reinterpret_cast<uintptr_t>(o) & 3) == 0) *reinterpret_cast<__half2*>(o) = __halves2half2(h0, h1);
            else { o[0] = h0; o[1] = h1; }
            if (RADII) { mean[which * D + c] = __half2float(h0); mean[which * D + c + 1] = __half2float(h1); }
        }
    } else if (tid < 2 * D) {
        const int which = tid / D, d = tid - which * D;
        float s = 0.f;
#pragma unroll 4
        for (int t = 0; t < kP; ++t) s = __fadd_rn(s, staged1<D>(src, which, t, d));
        const __half h = __float2half_rn(__fdiv_rn(s, (float)kP));
        reinterpret_cast<__half*>(j.dst + (which ? half_bytes(1, D) : 0))[d] = h;
        if (RADII) mean[which * D + d] = __half2float(h);
    }
    if constexpr (RADII) {
        work_sync();
        const int t = tid >> 2, q4 = tid & 3;
        const int f = NO == 4 ? (lane >> 1) & 3 : (lane >> 2) & 1;
        float top[2];
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            float e2 = 0.f;
#pragma unroll 1
            for (int o = 0; o < NO; ++o) {
                const int c8 = q4 * NO + (o ^ f);
                float x[8];
                staged_octet<D, SRC>(src, which, t, c8, x);
                const float4 a = *reinterpret_cast<const float4*>(mean + which * D + 8 * c8);
                const float4 b = *reinterpret_cast<const float4*>(mean + which * D + 8 * c8 + 4);
                const float mu[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int c = 0; c < 8; ++c) { const float e = __fsub_rn(x[c], mu[c]); e2 = fmaf(e, e, e2); }
            }
            e2 += __shfl_xor_sync(0xffffffffu, e2, 1);
            e2 += __shfl_xor_sync(0xffffffffu, e2, 2);
            top[which] = e2 == e2 ? e2 : 0.f;              // a token that is not a number counts as nothing, as in fmaxf
#pragma unroll
            for (int o = 16; o >= 4; o >>= 1) top[which] = fmaxf(top[which], __shfl_xor_sync(0xffffffffu, top[which], o));
        }
        if (lane == 0) { atomicMax(&sm.err[0], __float_as_uint(top[0])); atomicMax(&sm.err[1], __float_as_uint(top[1])); }
        work_sync();
        if (tid < 2) {
            float* acc = tid ? j.ev : j.ek;
            *acc += sqrtf(__uint_as_float(sm.err[tid]));
        }
    }
}

// The rungs of a source kind: PACKED launches demote (bf16 tiles of a rung-16 block, or a quantised block, which
// only moves further down), the others pack dense bf16 / fp16 rows.  MAY_RADII: the launch may ask for error radii.
template <int D, int SRC, bool RADII>
__device__ __forceinline__ void quantise_rung(const StagedSrc& src, const Job& j, Work& sm) {
    if (j.level == 1) { centroid_staged<D, SRC, RADII>(src, j, sm); return; }
    // one body per rung, so that every shift, mask and byte offset is a constant
    if constexpr (SRC != 3) {
        if (j.level == 8) { quantise_staged<D, 8, SRC, RADII>(src, j, sm); return; }
    }
    if (j.level == 4) quantise_staged<D, 4, SRC, RADII>(src, j, sm);
    else quantise_staged<D, 2, SRC, RADII>(src, j, sm);
}
template <int D, int SRC, bool MAY_RADII>
__device__ __forceinline__ void quantise_src(const StagedSrc& src, const Job& j, Work& sm) {
    if constexpr (MAY_RADII) {
        if (j.ek != nullptr) { quantise_rung<D, SRC, true>(src, j, sm); return; }
    }
    quantise_rung<D, SRC, false>(src, j, sm);
}

template <int D, bool PACKED, bool MAY_RADII>
__device__ void requantise_staged(const StagedSrc& src, const Job& j, Work& sm) {
    constexpr int OPR = D / 8, ROWS = kThreads / OPR, NI = kP / ROWS;
    const int tid = threadIdx.x;
    const int c8 = tid % OPR, tr = tid / OPR;
    const int lv = j.level;
    const int G = kP >> src.kgs, gv = D >> src.vgs;
    const bool quant = lv == 8 || lv == 4 || lv == 2;

    if (tid < 2) sm.err[tid] = 0u;
    if (!quant && j.zero_scales) {
        for (int u = tid; u < G * D; u += kThreads) { j.klo[u] = __ushort_as_half(0); j.kstep[u] = __ushort_as_half(0); }
        for (int u = tid; u < kP * gv; u += kThreads) { j.vlo[u] = __ushort_as_half(0); j.vstep[u] = __ushort_as_half(0); }
    }

    if (lv == 16) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            uint16_t* half = reinterpret_cast<uint16_t*>(j.dst + (w ? half_bytes(16, D) : 0));
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                float x[8];
                staged8<D>(src, w, tr + i * ROWS, c8, x);
                uint32_t o[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(x[2 * c], x[2 * c + 1]);
                    o[c] = *reinterpret_cast<const uint32_t*>(&b);
                }
                uint16_t* p = half + (size_t)(tr + i * ROWS) * D + 8 * c8;
                if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2], o[3]);
                else for (int c = 0; c < 4; ++c) { p[2 * c] = (uint16_t)o[c]; p[2 * c + 1] = (uint16_t)(o[c] >> 16); }
            }
        }
        return;
    }

    if constexpr (PACKED) {
        if (src.kind == 3) quantise_src<D, 3, MAY_RADII>(src, j, sm);
        else quantise_src<D, 1, MAY_RADII>(src, j, sm);
    } else {
        if (src.kind == 2) quantise_src<D, 2, MAY_RADII>(src, j, sm);
        else quantise_src<D, 1, MAY_RADII>(src, j, sm);
    }
}

}  // namespace rq
}  // namespace gkv
