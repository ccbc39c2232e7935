// shortlist.cuh — device helpers shared by the shortlist kernels: tcgen05
// descriptors and TMEM loads, bounded waits, the per-pair error bound, the
// certified comparisons, the work queues and the exact spec-order distance.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "ptx.cuh"
#include "slm_shortlist.h"

namespace slm {

// Order-preserving map of f32 to u32 (unsigned order == float order).
SLM_DEV uint32_t f2ord(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
SLM_DEV float ord2f(uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

SLM_DEV float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

SLM_DEV float warp_min_f32(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

SLM_DEV uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

typedef unsigned long long u64x;
SLM_DEV u64x f2_pack(float lo, float hi) {
    u64x d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
SLM_DEV float f2_lo(u64x v) { return __uint_as_float(static_cast<uint32_t>(v)); }
SLM_DEV float f2_hi(u64x v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
SLM_DEV u64x f2_sub(u64x a, u64x b) {
    u64x d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// 32 lanes x 16 consecutive 32-bit TMEM columns (asynchronous until the wait).
SLM_DEV void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// Waits for this thread's TMEM loads; the registers are operands so no use
// of them can be scheduled before the wait.
SLM_DEV void tmem_wait_ld16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                   "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                   "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

// Ties registers already waited for to this point, as tmem_wait_ld16 does.
SLM_DEV void tmem_tie16(uint32_t (&r)[16]) {
    asm volatile(""
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                   "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                   "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

// Merges another set's (smallest, second smallest, where) into this one's.
SLM_DEV void top2_merge(float &m1, float &m2, uint32_t &j, float o1, float o2, uint32_t oj) {
    m2 = min3f(m2, o2, fmaxf(m1, o1));
    j = o1 < m1 ? oj : j;
    m1 = fminf(m1, o1);
}

// ------------------------------------------------------------ tcgen05 pieces

// Shared-memory matrix descriptor (tcgen05): K-major, 128B swizzle, 8-row
// groups 1024 bytes apart (stride byte offset), version 1, base offset 0.
SLM_DEV uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fffu);   // start address
    d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset
    d |= (uint64_t)1 << 46;                    // descriptor version
    d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
    return d;
}

// Shared-memory matrix descriptor: K-major without swizzle. Core matrices of
// 8 rows x 16 bytes (rows 16 bytes apart); lbo = bytes between core matrices
// along K, sbo = bytes between 8-row groups.
SLM_DEV uint64_t umma_desc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fffu);
    d |= (uint64_t)((lbo >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3fffu) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version; layout type 0 = no swizzle
    return d;
}

// Instruction descriptor: kind::f8f6f4 with e4m3 inputs (format 0), f32
// accumulate, K-major A and B, M=128, N=128.
__host__ __device__ constexpr uint32_t fp8_idesc() { return (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24); }

// Bounded wait (about 2 s of wall time); on timeout raises the CTA abort flag
// and records an error so every role leaves its loop.
SLM_DEV bool sl_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag, uint32_t *err) {
    uint64_t t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63) == 63) {
            if (*abort_flag) return false;
            const uint64_t now = globaltimer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > 2000000000ull) {
                *abort_flag = 1;
                atomicCAS(err, 0u, (uint32_t)DERR_TIMEOUT_MMA);
                return false;
            }
        }
    }
}

// The loads into a ring of `stages` (`issued` were started in all) land before the CTA
// ends, also when a wait gave up and nobody took them. Bounded like that wait.
SLM_DEV void drain_loads(uint64_t *full, uint32_t stages, uint32_t issued) {
    for (uint32_t q = 0; q < stages && q < issued; ++q)
        mbar_wait(&full[(issued - 1 - q) % stages], ((issued - 1 - q) / stages) & 1, nullptr);
}

// ------------------------------------------------------------ error bound

// The per-pair error bound of this launch's precision (g.fp8) from the two
// views' statistics; false when the pair cannot be certified (non-finite or
// huge inputs).
SLM_DEV bool pair_eps(const SlArgs &g, const SlPair &sp, float *eps_out) {
    const ViewStat va = g.vstats[sp.view_a], vb = g.vstats[sp.view_b];
    const double A = __uint_as_float(va.nmax), B = __uint_as_float(vb.nmax);
    const double Ra = __uint_as_float(va.rho), Rb = __uint_as_float(vb.rho);
    const double Qa = __uint_as_float(va.nqmax), Qb = __uint_as_float(vb.nqmax);
    bool unsafe = va.bad || vb.bad || !(A <= 64.0) || !(B <= 64.0);
    // |d~ - d| <= 2 |a.b - q(a).q(b)| + accumulation and rounding terms, with
    // |a.b - q(a).q(b)| <= |a - q(a)| |b| + |q(a)| |b - q(b)| (Cauchy-Schwarz).
    double eps = 2.0 * (Ra * B + Qa * Rb) * (1.0 + 1e-3);
    eps += 5e-4 * Qa * Qb + 5e-5 * (A * A + B * B) + 2e-5 * (A + B) * (A + B) + 1e-6;
    // BF16: the tensor core also accumulates the folded norms (|a|^2 + |b|^2) / 2
    // and their bf16 split (relative 2^-17); the accumulation is taken as no
    // better than 2^-11 relative to that magnitude, doubled with d~
    if (!g.fp8) eps += 5e-4 * (A * A + B * B);
    if (!(eps < 1e30)) unsafe = true;
    *eps_out = unsafe ? __int_as_float(0x7f800000) : (float)(eps * (1.0 + 1e-6));
    return !unsafe;
}

// ------------------------------------------------------- certified tests

// The decisions below are proved in f32 with directed rounding: each side of
// a comparison is rounded toward the weaker claim, so a true comparison of the
// rounded values implies it for the real numbers. The factors cover the
// reference's own rounding of (r*r)*d2 (at most 2^-24 relative).
constexpr float kUp = 1.000001f;    // > 1 + 2^-24
constexpr float kDown = 0.999999f;  // < 1 - 2^-24

// No match for the row: d1 >= m1 - eps >= r^2 (m2 + eps) kUp >= fl(r^2 d2),
// where m1 - eps bounds d1 from below and m2 + eps bounds d2 from above.
SLM_DEV bool certain_no_match(float m1, float m2, float eps, float r2) {
    return __fsub_rd(m1, eps) >= __fmul_ru(__fmul_ru(r2, __fadd_ru(m2, eps)), kUp);
}

// The ratio test passes: d1 <= a1 + eps < r^2 (a2 - eps) kDown <= fl(r^2 d2).
SLM_DEV bool certain_ratio_pass(float a1, float a2, float eps, float r2) {
    return __fadd_ru(a1, eps) < __fmul_rd(__fmul_rd(r2, __fsub_rd(a2, eps)), kDown);
}

// Window x + 2 eps, rounded up (a larger threshold only admits more); NaN
// becomes +inf (admit everything).
SLM_DEV float window_up(float x, float eps) {
    const float t = __fmul_ru(__fadd_ru(x, 2.f * eps), kUp);
    return t == t ? t : __int_as_float(0x7f800000);
}

// Row blocks of a pair: enough for its rows and its columns.
SLM_DEV uint32_t pair_blocks(const PairMeta &pm) {
    const uint32_t n = max(pm.na, pm.nb);
    return max(1u, (n + kSlRowBlock - 1) / kSlRowBlock);
}

// ------------------------------------------------------------ exact work

SLM_DEV void sl_push(SlQueue *q, uint32_t *len, uint32_t cap, uint32_t *err, uint32_t pair, uint32_t kind, uint32_t i,
                     uint32_t j) {
    const uint32_t s = atomicAdd(len, 1u);
    if (s < cap) {
        SlQueue e;
        e.pair = pair;
        e.kind = kind;
        e.i = i;
        e.j = j;
        q[s] = e;
    } else {
        atomicCAS(err, 0u, (uint32_t)DERR_BAD_ITEM);
    }
}

SLM_DEV void push_scan(const SlArgs &g, uint32_t pair, uint32_t kind, uint32_t i, uint32_t j) {
    sl_push(g.queue, &g.ctl[kCtlScanLen], g.queue_cap, g.ctl + 1, pair, kind, i, j);
}

// Exact distance by 8 lanes: lane k of the group accumulates components
// 8c+k for c = 0..15 (matching.rs:146-155), then the lane sums are added in
// order 0..7. p and r may differ per group; the result is valid in all 8 lanes.
SLM_DEV float dist8(const float *__restrict__ p, const float *__restrict__ r) {
    const uint32_t lane = threadIdx.x & 31, k = lane & 7, base = lane & ~7u;
    float acc = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const float t = __fsub_rn(p[8 * c + k], r[8 * c + k]);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
    }
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) s = __fadd_rn(s, __shfl_sync(0xffffffffu, acc, base + q));
    return s;
}

// The same from one row to many: the row's share of a lane (components 8c + k) is kept.
SLM_DEV void load8(const float *p, float (&own)[16]) {
#pragma unroll
    for (int c = 0; c < 16; ++c) own[c] = p[8 * c + (threadIdx.x & 7)];
}
SLM_DEV float dist8(const float (&own)[16], const float (&other)[16]) {
    const uint32_t base = threadIdx.x & 24;  // the group's first lane
    float acc = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const float t = __fsub_rn(own[c], other[c]);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
    }
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) s = __fadd_rn(s, __shfl_sync(0xffffffffu, acc, base + q));
    return s;
}

// The same by 2 lanes, 16 distances a warp: lane h of a pair holds the sums of
// components 8c + 4h .. 8c + 4h + 3; the even lane adds its four in order and
// hands the sum to the odd lane, which adds its own. p and r (16-byte aligned)
// may differ per pair of lanes; the result is valid in both.
template <int U = 16>
SLM_DEV float dist2(const float *__restrict__ p, const float *__restrict__ r) {
    const uint32_t h = threadIdx.x & 1;
    const float4 *p4 = reinterpret_cast<const float4 *>(p) + h, *r4 = reinterpret_cast<const float4 *>(r) + h;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll U
    for (int c = 0; c < 16; ++c) {
        const float4 x = p4[2 * c], y = r4[2 * c];
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float t = __fsub_rn(xs[k], ys[k]);
            acc[k] = __fadd_rn(acc[k], __fmul_rn(t, t));
        }
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) s = __fadd_rn(s, acc[k]);
    float u = __shfl_xor_sync(0xffffffffu, s, 1);  // the odd lane gets the even lane's sum
#pragma unroll
    for (int k = 0; k < 4; ++k) u = __fadd_rn(u, acc[k]);
    return __shfl_sync(0xffffffffu, u, (threadIdx.x & 31) | 1);
}

}  // namespace slm
