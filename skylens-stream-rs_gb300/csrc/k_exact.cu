// k_exact.cu — the plain FP32 matcher (exact, bit-identical to the reference).
//
// Reference: crates/core/src/matching.rs:144-215 (sq_dist + ratio_match).
//
// Layout. Descriptors live in store tiles of 128 rows: tile[slot][row] with
// slot = perm_slot(k) = (k % 8) * 16 + k / 8, so walking slots 0..127 walks
// sq_dist's order: lane 0 (components 0, 8, ..., 120), then lane 1, and so
// on. One walk of 16 slots is one lane accumulator; the 8 lane sums are added
// to the distance in lane order. Every operation is an explicit _rn IEEE op
// (no FMA contraction), so each d(i, j) equals the reference's f32 value.
//
// Kernel. A persistent CTA (eight computing warps and one that loads, one CTA per
// SM) takes work items (a 128-row tile of a, or some of its groups of 32 rows,
// against a range of b's groups of 32 columns) from a global counter. The a tile is bulk-copied (TMA) into shared memory
// once per item; b tiles stream in halves through a four-slot TMA/mbarrier ring.
// Each thread owns an 8 x 8 register block of distances: two neighbouring rows
// and columns in each group of 32 (row_of, col_of).
//   rows:    best / second-best / argmin are carried in registers across the
//            b tiles and merged across the 16 column threads at the end of
//            the item with warp shuffles (order-independent: min, lowest j on
//            ties, second smallest of the multiset).
//   columns: (bits(d) << 32 | i) keys are min-reduced in the warp, then with one
//            global atomicMin per column, warp and tile; unsigned order of the
//            key is (d, lowest i) because d >= +0.
// The finalize kernel merges row partials, applies the ratio test
// (d1 < (r*r)*d2 in f32) and the mutual check, and compacts in ascending i.
#include <cuda_runtime.h>

#include <type_traits>

#include "pack.cuh"
#include "ptx.cuh"
#include "slm_internal.h"

namespace slm {

// ------------------------------------------------------------------ pack

// Many views at once: one CTA per 32-row group (blockIdx.y) of each entry of
// a tile table {first row-major row, rows from it on, store tile, view}.
__global__ void __launch_bounds__(256) pack_fp32_tiles_kernel(const uint4 *__restrict__ tab,
                                                              const float *__restrict__ raw,
                                                              float *__restrict__ tiled) {
    __shared__ float sm[32][kDesc + 1];
    const uint4 e = tab[blockIdx.x];
    pack_group(raw + (size_t)e.x * kDesc, e.y, tiled + (size_t)e.z * kTileFloats, 0u, blockIdx.y, sm);
}

void launch_pack_fp32_tiles(const uint4 *tab, uint32_t ntiles, const float *raw, float *tiled, cudaStream_t s) {
    if (ntiles) pack_fp32_tiles_kernel<<<dim3(ntiles, 4), 256, 0, s>>>(tab, raw, tiled);
}

__global__ void fill_u64_kernel(unsigned long long *p, uint64_t n, unsigned long long v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

void launch_fill_u64(unsigned long long *p, uint64_t n, unsigned long long v, cudaStream_t s) {
    if (!n) return;
    uint64_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    fill_u64_kernel<<<(unsigned)blocks, 256, 0, s>>>(p, n, v);
}

// ----------------------------------------------------------- exact match

constexpr int kWarps = 8;                        // each 16 of a tile's rows against its 128 columns
constexpr int kThreads = 32 * (kWarps + 4);      // and a group of four, of which one loads
// Registers a thread: 168 at launch (504 a lane for the three warps of a
// scheduler), the loading group's given to the two computing warps: 40 + 2 x 232.
constexpr int kLoadRegs = 40, kComputeRegs = 232;
static_assert(kLoadRegs + 2 * kComputeRegs <= 3 * 168 && 3 * 168 * 32 <= 16384, "registers of a scheduler");
constexpr int kRing = 4;                         // halves of b tiles in flight
constexpr uint32_t kHalfFloats = kTileFloats / 2;  // 64 of the 128 dimensions
constexpr uint32_t kHalfBytes = kHalfFloats * 4;
constexpr int kUnroll = 5;
constexpr uint32_t kNoItem = 0xffffffffu;

struct ExactSmem {
    float A[2][kHalfFloats];
    float B[kRing][kHalfFloats];
    uint64_t fullA[2], emptyA[2], fullB[kRing], emptyB[kRing];
    Item item[2];
    PairMeta pm[2];
};

typedef unsigned long long u64;

SLM_DEV u64 f2_sub(u64 a, u64 b) {
    u64 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
SLM_DEV u64 f2_add(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
SLM_DEV u64 f2_fma(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
SLM_DEV u64 f2_pack(float lo, float hi) {
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
SLM_DEV float f2_lo(u64 v) { return __uint_as_float(static_cast<uint32_t>(v)); }
SLM_DEV float f2_hi(u64 v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }

// A thread's rows and columns of a tile: two neighbours in each 32 (group q).
SLM_DEV int row_of(int ty, int r) { return 32 * (r >> 1) + 2 * ty + (r & 1); }
SLM_DEV int col_of(int tx, int c) { return 32 * (c >> 1) + 2 * tx + (c & 1); }

// Half of the spec-order distances' sums between the thread's rows and columns
// (tile halves in [slot][row] layout), in the first NR row and NC column groups:
// lanes 0..3 or 4..7 of the reference's eight partial sums, added to s in order.
template <bool X2, int NR, int NC>
SLM_DEV void half_distances(const float *sa, const float *sb, int ty, int tx, u64 zero2, u64 (&s)[8][4]) {
#pragma unroll 1
    for (int lane = 0; lane < 4; ++lane) {
        u64 acc[8][4];
        const float *pa = sa + lane * 16 * kTile + 2 * ty;
        const float *pb = sb + lane * 16 * kTile + 2 * tx;
        const auto step = [&](auto first) {
            float av[2 * NR];
            u64 bv[NC];
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                const float2 v = *reinterpret_cast<const float2 *>(pa + 32 * q);
                av[2 * q] = v.x;
                av[2 * q + 1] = v.y;
            }
#pragma unroll
            for (int q = 0; q < NC; ++q) bv[q] = *reinterpret_cast<const u64 *>(pb + 32 * q);
            pa += kTile;
            pb += kTile;
#pragma unroll
            for (int r = 0; r < 2 * NR; ++r) {
                if constexpr (X2) {
                    // Packed pairs of columns: {a_r, a_r} - {b_c, b_c+1}. A packed
                    // multiply followed by a packed add is contracted to a packed FMA by
                    // the code generator (measured: 25 % of distances off by an ulp). The
                    // square is therefore a packed FMA t * t + z with z a run-time zero (a
                    // kernel argument the compiler cannot fold): rounded once, it is
                    // exactly RN(t * t) (t * t >= 0, + 0 changes nothing), and no
                    // contraction with the following add is possible.
                    const u64 ar = f2_pack(av[r], av[r]);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const u64 t = f2_sub(ar, bv[c]);
                        const u64 tt = f2_fma(t, t, zero2);
                        acc[r][c] = decltype(first)::value ? tt : f2_add(acc[r][c], tt);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const float t0 = __fsub_rn(av[r], f2_lo(bv[c])), t1 = __fsub_rn(av[r], f2_hi(bv[c]));
                        const float q0 = __fmul_rn(t0, t0), q1 = __fmul_rn(t1, t1);
                        acc[r][c] = decltype(first)::value
                                        ? f2_pack(q0, q1)
                                        : f2_pack(__fadd_rn(f2_lo(acc[r][c]), q0), __fadd_rn(f2_hi(acc[r][c]), q1));
                    }
                }
            }
        };
        step(std::true_type{});
        // (all 15 unrolled, the code of warps out of step outgrows the instruction
        // caches: 13.2 ms for the 60 views below; 3 at a time 11.1, 5 at a time 11.0)
#pragma unroll kUnroll
        for (int c16 = 1; c16 < 16; ++c16) step(std::false_type{});
#pragma unroll
        for (int r = 0; r < 2 * NR; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c)
                s[r][c] = X2 ? f2_add(s[r][c], acc[r][c])
                             : f2_pack(__fadd_rn(f2_lo(s[r][c]), f2_lo(acc[r][c])),
                                       __fadd_rn(f2_hi(s[r][c]), f2_hi(acc[r][c])));
    }
}

// What a consumer warp carries through an item.
struct ExactWarp {
    const ExactArgs &g;
    ExactSmem &S;
    int tx, ty, lane;
    u64 zero2;
    uint32_t seq;  // halves of b tiles consumed: ring slot and parity
    uint32_t a1;   // second halves of a tiles consumed
    float d1[8], d2[8];
    uint32_t j1[8];
};

// One b tile: its distances in two halves, then ratio_match's row update and the
// column minima. CHECK: the tile's last row and column groups are not whole.
// False when a bounded wait gave up.
template <bool X2, int NR, int NC, bool CHECK>
SLM_DEV bool exact_tile(ExactWarp &w, const PairMeta &pm, uint32_t row0, uint32_t col0, bool first, bool last) {
    ExactSmem &S = w.S;
    u64 s[8][4];
#pragma unroll
    for (int r = 0; r < 2 * NR; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) s[r][c] = 0ull;
#pragma unroll 1
    for (int h = 0; h < 2; ++h, ++w.seq) {
        const uint32_t slot = w.seq % kRing;
        // (the item's first half was waited for before the item was read)
        bool ok = !first || h == 0 || mbar_wait(&S.fullA[1], w.a1 & 1, w.g.err);
        ok = ok && mbar_wait(&S.fullB[slot], (w.seq / kRing) & 1, w.g.err);
        if (!__all_sync(0xffffffffu, ok)) return false;
        half_distances<X2, NR, NC>(S.A[h] + row0 % kTile, S.B[slot] + col0 % kTile, w.ty, w.tx, w.zero2, s);
        __syncwarp();
        if (w.lane == 0) {
            mbar_arrive(&S.emptyB[slot]);
            if (last) mbar_arrive(&S.emptyA[h]);
        }
    }
    float d[2 * NR][2 * NC];
#pragma unroll
    for (int r = 0; r < 2 * NR; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            d[r][2 * c] = f2_lo(s[r][c]);
            d[r][2 * c + 1] = f2_hi(s[r][c]);
        }
    // rows: ratio_match's update (matching.rs:182-187), columns in increasing j;
    // a NaN changes nothing (fminf takes the other operand)
#pragma unroll
    for (int c = 0; c < 2 * NC; ++c) {
        const uint32_t j = col0 + col_of(w.tx, c);
        if (CHECK && c >= 2 * NC - 2 && j >= pm.nb) break;
#pragma unroll
        for (int r = 0; r < 2 * NR; ++r) {
            const float v = d[r][c];
            const bool less = v < w.d1[r];
            const float other = fminf(w.d2[r], v);
            w.d2[r] = less ? w.d1[r] : other;
            w.d1[r] = fminf(w.d1[r], v);
            w.j1[r] = less ? j : w.j1[r];
        }
    }
    // columns: (d, lowest i) (matching.rs:188-190, 196-203). Only finite minima
    // matter: a row's best column always holds one.
    if (w.g.mutual) {
        u64 key[2 * NC];
#pragma unroll
        for (int c = 0; c < 2 * NC; ++c) {
            float best = __int_as_float(0x7f800000);
            uint32_t at = 0xffffffffu;
#pragma unroll
            for (int r = 0; r < 2 * NR; ++r) {
                const uint32_t i = row0 + row_of(w.ty, r);
                if (d[r][c] < best && !(CHECK && r >= 2 * NR - 2 && i >= pm.na)) {
                    best = d[r][c];
                    at = i;
                }
            }
            key[c] = (u64)__float_as_uint(best) << 32 | at;
            const u64 o = __shfl_xor_sync(0xffffffffu, key[c], 16);
            key[c] = o < key[c] ? o : key[c];
        }
        // the even columns by one half warp, the odd ones by the other
#pragma unroll
        for (int c = 0; c < 2 * NC; c += 2) {
            const u64 k = w.lane < 16 ? key[c] : key[c + 1];
            const uint32_t j = col0 + col_of(w.tx, c) + (w.lane >> 4);
            if ((uint32_t)k != 0xffffffffu && (!CHECK || j < pm.nb)) atomicMin(&w.g.colbest[pm.col_base + j], k);
        }
    }
    return true;
}

template <bool X2, int NR>
SLM_DEV bool exact_edge(uint32_t nc, ExactWarp &w, const PairMeta &pm, uint32_t row0, uint32_t col0, bool first,
                        bool last) {
    switch (nc) {
        case 1: return exact_tile<X2, NR, 1, true>(w, pm, row0, col0, first, last);
        case 2: return exact_tile<X2, NR, 2, true>(w, pm, row0, col0, first, last);
        case 3: return exact_tile<X2, NR, 3, true>(w, pm, row0, col0, first, last);
        default: return exact_tile<X2, NR, 4, true>(w, pm, row0, col0, first, last);
    }
}

// Persistent: a warp that loads and eight that compute, which meet only at the
// tiles' mbarriers. Bound by the FP32 pipe (three operations per dimension and
// distance, a packed one every other clock): the row and column updates are ALU
// work, and a warp's run behind the others' distances as long as no barrier ties
// the warps together, so the halves of the tiles are released one by one, a ring
// of four holds the next, and column minima go straight to the pair's (a shared
// reduction needed a barrier a tile). Views are rarely whole tiles: the last row
// and column tile of a pair compute only the groups of 32 that hold any.
// 60 views' pairs of about 1150 x 1150 rows: 12.6 ms with a barrier a tile and
// whole tiles (77 % of the pipe counting real distances), now 11.0 (90 %); one pair
// of 317 x 300 rows 57.5 us before, now 54.5.
template <bool X2>
__global__ void __launch_bounds__(kThreads, 1) exact_kernel(ExactArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    ExactSmem &S = *reinterpret_cast<ExactSmem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int h = 0; h < 2; ++h) {
            mbar_init(&S.fullA[h], 1);
            mbar_init(&S.emptyA[h], kWarps);
        }
        for (int q = 0; q < kRing; ++q) {
            mbar_init(&S.fullB[q], 1);
            mbar_init(&S.emptyB[q], kWarps);
        }
        fence_mbar_init();
    }
    __syncthreads();
    grid_wait();
    // Items planned on the device (pairs routed from the shortlist path) come
    // with their count in device memory, written by an earlier kernel.
    const uint32_t n_items = g.n_items_dev ? min(*g.n_items_dev, g.n_items) : g.n_items;
    if (warp >= kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLoadRegs));
        if (tid == 32 * kWarps) {
            uint32_t k = 0, seq = 0, a0 = 0, a1 = 0;  // items; halves of b and of a tiles loaded so far
            bool ok = true;
            for (;; ++k) {
                const uint32_t it = atomicAdd(g.work, 1u);
                // every warp is done with the a tile's first half, so with the item before its own
                ok = k == 0 || mbar_wait(&S.emptyA[0], (k - 1) & 1, g.err);
                if (!ok) break;
                if (it >= n_items) {
                    S.item[k & 1].pair = kNoItem;
                    mbar_arrive(&S.fullA[0]);
                    break;
                }
                const Item item = g.items[it];
                const PairMeta pm = g.pairs[item.pair];
                S.item[k & 1] = item;
                S.pm[k & 1] = pm;
                const float *at = g.tiled + (size_t)(pm.a_row0 / kTile + item.rt) * kTileFloats;
                const float *bt = g.tiled + (size_t)(pm.b_row0 / kTile + item.q0 / 4) * kTileFloats;
                const uint32_t nh = item.q0 < item.q1 ? 2 * ((item.q1 + 3) / 4 - item.q0 / 4) : 0;
                mbar_arrive_expect_tx(&S.fullA[0], kHalfBytes);
                bulk_g2s(S.A[0], at, kHalfBytes, &S.fullA[0]);
                ++a0;
                for (uint32_t q = 0; q < nh && ok; ++q, ++seq) {
                    const uint32_t slot = seq % kRing, use = seq / kRing;
                    ok = use == 0 || mbar_wait(&S.emptyB[slot], (use - 1) & 1, g.err);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&S.fullB[slot], kHalfBytes);
                    bulk_g2s(S.B[slot], bt + (size_t)q * kHalfFloats, kHalfBytes, &S.fullB[slot]);
                    if (q == 0) {
                        ok = a1 == 0 || mbar_wait(&S.emptyA[1], (a1 - 1) & 1, g.err);
                        if (!ok) {
                            ++seq;
                            break;
                        }
                        mbar_arrive_expect_tx(&S.fullA[1], kHalfBytes);
                        bulk_g2s(S.A[1], at + kHalfFloats, kHalfBytes, &S.fullA[1]);
                        ++a1;
                    }
                }
                if (!ok) break;
            }
            if (!ok) {  // a wait gave up: no copy may be in flight when the CTA ends
                if (a0) mbar_wait(&S.fullA[0], (a0 - 1) & 1, g.err);
                if (a1) mbar_wait(&S.fullA[1], (a1 - 1) & 1, g.err);
                for (uint32_t q = 0; q < kRing; ++q)
                    if (seq > q) mbar_wait(&S.fullB[q], ((seq - 1 - q) / kRing) & 1, g.err);
            }
        }
        __syncwarp();
        __syncthreads();
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kComputeRegs));
    ExactWarp w{g, S, lane & 15, tid >> 4, lane, f2_pack(g.zero, g.zero), 0u, 0u, {}, {}, {}};
    for (uint32_t k = 0;; ++k) {
        if (!__all_sync(0xffffffffu, mbar_wait(&S.fullA[0], k & 1, g.err))) break;
        const Item item = S.item[k & 1];
        if (item.pair == kNoItem) break;
        const PairMeta pm = S.pm[k & 1];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            w.d1[r] = __int_as_float(0x7f800000);
            w.d2[r] = __int_as_float(0x7f800000);
            w.j1[r] = 0xffffffffu;
        }
        const uint32_t row0 = item.rt * kTile + 32 * item.g0, nr = min((pm.na - row0 + 31) / 32, item.g1 - item.g0);
        bool ok = true;
        for (uint32_t q = item.q0, end; q < item.q1 && ok; q = end) {
            end = min(q / 4 * 4 + 4, item.q1);  // of this tile's groups
            const uint32_t col0 = 32 * q, nc = end - q;
            const bool first = q == item.q0, last = end == item.q1;
            if (nr == 4 && nc == 4 && row0 + kTile <= pm.na && col0 + kTile <= pm.nb)
                ok = exact_tile<X2, 4, 4, false>(w, pm, row0, col0, first, last);
            else if (nr == 1)
                ok = exact_edge<X2, 1>(nc, w, pm, row0, col0, first, last);
            else if (nr == 2)
                ok = exact_edge<X2, 2>(nc, w, pm, row0, col0, first, last);
            else if (nr == 3)
                ok = exact_edge<X2, 3>(nc, w, pm, row0, col0, first, last);
            else
                ok = exact_edge<X2, 4>(nc, w, pm, row0, col0, first, last);
        }
        if (!ok) break;
        if (item.q0 < item.q1) {
            ++w.a1;
        } else {  // no b tiles, and no second half of the a tile was loaded
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.emptyA[0]);
        }
        // Merge row states across the 16 column threads (lanes xor 1..8).
#pragma unroll
        for (int r = 0; r < 8; ++r) {
#pragma unroll
            for (int off = 1; off < 16; off <<= 1) {
                const float o1 = __shfl_xor_sync(0xffffffffu, w.d1[r], off);
                const float o2 = __shfl_xor_sync(0xffffffffu, w.d2[r], off);
                const uint32_t oj = __shfl_xor_sync(0xffffffffu, w.j1[r], off);
                const float nd2 = fminf(fmaxf(w.d1[r], o1), fminf(w.d2[r], o2));
                if (o1 < w.d1[r] || (o1 == w.d1[r] && oj < w.j1[r])) {
                    w.d1[r] = o1;
                    w.j1[r] = oj;
                }
                w.d2[r] = nd2;
            }
        }
        if (w.tx == 0) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                if ((uint32_t)r / 2 >= nr) break;  // other items' rows, or none
                RowPart p;
                p.d1 = w.d1[r];
                p.d2 = w.d2[r];
                p.j1 = w.j1[r];
                p.pad = 0;
                g.parts[(size_t)item.part * kTile + 32 * item.g0 + row_of(w.ty, r)] = p;
            }
        }
    }
    __syncthreads();
}

cudaError_t init_exact_kernels() {
    const int smem = (int)sizeof(ExactSmem);
    cudaError_t e = cudaFuncSetAttribute(exact_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(exact_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

void launch_exact(const ExactArgs &a, int grid, cudaStream_t s) {
    const size_t smem = sizeof(ExactSmem);
    launch_next(a.x2 ? exact_kernel<true> : exact_kernel<false>, grid, kThreads, smem, s, a);
}

// -------------------------------------------------------------- finalize

// One CTA per pair: merge the row partials of every column chunk, apply
// matching.rs:204-214 and write matches in ascending i. One thread per row and
// step, partials loaded four at a time: a batch of few pairs runs 1024 threads
// per pair, since a single small pair is a chain of dependent loads, not a
// bandwidth problem; larger batches run 256 (more pairs resident per SM).
constexpr int kFinThreadsMax = 1024;

template <int kThreads>
__global__ void __launch_bounds__(kThreads) finalize_kernel(FinalizeArgs g) {
    grid_wait();
    __shared__ uint32_t warp_tot[kThreads / 32];
    constexpr uint32_t nthr = kThreads;
    constexpr int nwarps = kThreads / 32;
    const PairMeta pm = g.pairs[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const float kInf = __int_as_float(0x7f800000);
    uint32_t base = 0;
    for (uint32_t row0 = 0; row0 < pm.na; row0 += nthr) {
        const uint32_t i = row0 + tid;
        uint32_t flag = 0, jout = 0;
        if (i < pm.na) {
            const uint32_t rt = i / kTile;
            float d1 = kInf, d2 = kInf;
            uint32_t j1 = 0xffffffffu;
            const RowPart *pr = g.parts + (size_t)(pm.part_base + rt * pm.nchunk) * kTile + (i % kTile);
            if constexpr (kThreads == 256) {  // many pairs: mostly one column range per row
                for (uint32_t c = 0; c < pm.nchunk; ++c) merge_rowpart(pr[(size_t)c * kTile], d1, d2, j1);
            } else
            for (uint32_t c0 = 0; c0 < pm.nchunk; c0 += 4) {
                RowPart q[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    // an absent chunk merges as the neutral partial (inf, inf, none)
                    q[u] = RowPart{kInf, kInf, 0xffffffffu, 0u};
                    if (c0 + u < pm.nchunk) q[u] = pr[(size_t)(c0 + u) * kTile];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) merge_rowpart(q[u], d1, d2, j1);
            }
            const bool d2_finite = d2 < kInf;
            if (j1 != 0xffffffffu && d2_finite && !(d1 >= __fmul_rn(g.ratio2, d2))) {
                if (!g.mutual || static_cast<uint32_t>(g.colbest[pm.col_base + j1]) == i) {
                    flag = 1;
                    jout = j1;
                }
            }
        }
        // Block-wide exclusive scan of the flags.
        const uint32_t ballot = __ballot_sync(0xffffffffu, flag);
        const uint32_t wpre = __popc(ballot & ((1u << lane) - 1u));
        if (lane == 0) warp_tot[wid] = __popc(ballot);
        __syncthreads();
        uint32_t off = 0, tot = 0;
        for (int w = 0; w < nwarps; ++w) {
            const uint32_t t = warp_tot[w];
            off += (w < wid) ? t : 0;
            tot += t;
        }
        if (flag) g.slots[pm.slot_off + base + off + wpre] = make_uint2(i, jout);
        base += tot;
        __syncthreads();
    }
    if (tid == 0) g.counts[blockIdx.x] = (g.err && *g.err) ? 0xffffffffu : base;
}

void launch_finalize(const FinalizeArgs &a, cudaStream_t s) {
    if (!a.npairs) return;
    if (a.npairs <= kFewPairs)
        launch_next(finalize_kernel<kFinThreadsMax>, a.npairs, kFinThreadsMax, 0, s, a);
    else
        launch_next(finalize_kernel<256>, a.npairs, 256, 0, s, a);
}

// Self-test of the bounded waits: thread 0 waits on an mbarrier that expects
// one arrival nobody makes, gives up after `polls` polls and records
// DERR_TIMEOUT_BAR in *err, the path every kernel's timed-out wait takes.
__global__ void wait_selftest_kernel(uint32_t polls, uint32_t *err) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_wait(&bar, 0, err, polls);
}

void launch_wait_selftest(uint32_t polls, uint32_t *err, cudaStream_t s) {
    wait_selftest_kernel<<<1, 32, 0, s>>>(polls, err);
}

}  // namespace slm
