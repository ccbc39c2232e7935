// k_top2.cu — the BF16 shortlist: one tensor-core pass per direction that
// leaves, for every row, its nearest column and its two smallest distance
// estimates; then the decisions they certify, and the rows they do not.
//
// Reference: crates/core/src/matching.rs:144-215. ratio_match needs a row's two
// smallest distances and its nearest column, and, for the cross-check, the
// nearest row of that column. Pass (a, b) gives the first for every row of a,
// pass (b, a) the second for every row of b; both are the same kernel.
//
// sl_top2_kernel (persistent, one CTA per SM, 18 warps):
//   warp 0      TMA producer: 1 or 2 a tiles of 128 rows, kept while
//               consecutive segments share them; b tiles two at a time (256
//               columns, 72 KiB) through two stages.
//   warp 1      one thread issues tcgen05.mma, M = 128, N = 256, K = 16: per a
//               tile 8 steps over the components (B negated) and one over the
//               norm extension, so the accumulator is d~ / 2. Two accumulators
//               of 256 TMEM columns take turns.
//   warps 2-17  epilogue: warp w reads TMEM lane quarter w % 4, every fourth
//               16-column chunk, one thread per row.
// What a row keeps, exactly, at 13 instructions per 16 columns:
//   - the minimum of each chunk comes with the load (tcgen05.ld.red); running
//     best, second best and best chunk of these minima;
//   - the running minimum of each of the 16 column classes (column mod 16).
//   The best column is (best chunk, best class). The second smallest distance
//   lies in another chunk or, if in the same, in another class: it is the
//   smaller of the second best chunk minimum and the second best class
//   minimum. (Equal minima give a second best equal to the best, which
//   certifies nothing, so their column does not matter.)
//
// Why this shape. N = 256: with N = 128 every MMA reads as many bytes of A as
// of B from shared memory, 128 bytes per clock for 64 clocks of tensor work;
// N = 256 reads 12 KiB per 128 clocks. A second pass in the other direction
// costs one more run over the tensor cores, but rows only: minima over the 32
// lanes of a warp (redux) for the column side took more issue slots than the
// whole row epilogue does. The epilogue takes 29 clocks per 32 x 16 chunk and
// sub-partition (measured alone; 43 with a min tree instead of ld.red) where
// the MMA takes 72, so the tensor pipe is the bound: 1.73 ms for both
// directions of a 240-view zone (3663 pairs, 2 x 4.87 G distances), 94 % of the
// measured BF16 rate with the padding of ragged tiles counted. The two passes
// before (N = 128; row and column minima, then the candidates of each row
// recomputed against a threshold) took 1.33 and 1.64 ms, and the zone's batch
// with its lists read back 3.50 ms; now 2.07.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "shortlist.cuh"

namespace slm {

namespace {

constexpr uint32_t kKb = 16384;                              // one K block (64 components) of a 128-row tile
constexpr uint32_t kStageBytes = 2 * kBf16TileStride;        // two b tiles, K block by K block
constexpr uint32_t kStageExt = 4 * kKb;                      // their norm extensions, after the four K blocks
constexpr int kTopStages = 2;
static_assert(kStageExt + 2 * kBf16ExtBytes == kStageBytes, "stage layout");

struct TopSmem {
    uint8_t A[2][kBf16TileStride];
    uint8_t B[kTopStages][kStageBytes];
    float2 mm[2][3][128];  // [a tile][other column group][row]: (m1, m2) to merge
    uint32_t mj[2][3][128];
    uint64_t a_full, a_empty;
    uint64_t b_full[kTopStages], b_empty[kTopStages];
    uint64_t t_full[2], t_empty[2];
    uint32_t tmem_base;
    uint32_t abort_flag;
};
constexpr size_t kTopSmemBytes = sizeof(TopSmem) + 1024;  // slack for 1024-byte alignment
static_assert(kTopSmemBytes <= 232448, "shared memory of one CTA");

// 32 lanes x 16 TMEM columns and their minimum (asynchronous until the wait);
// NaN columns are ignored unless all 16 are NaN.
SLM_DEV void tmem_ld16_min(uint32_t taddr, uint32_t (&r)[16], uint32_t &mn) {
    asm volatile(
        "tcgen05.ld.red.sync.aligned.32x32b.x16.min.f32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, %16, [%17];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(mn)
        : "r"(taddr)
        : "memory");
}

// Per row of one a tile and column group, over a segment's columns.
struct RowTop {
    float cls[16];      // minimum of each column class
    float m1, m2;       // two smallest chunk minima
    uint32_t chunk;     // chunk of m1
    SLM_DEV void reset() {
        const float inf = __int_as_float(0x7f800000);
#pragma unroll
        for (int k = 0; k < 16; ++k) cls[k] = inf;
        m1 = m2 = inf;
        chunk = 0;
    }
    SLM_DEV void add_min(float cm, uint32_t c) {
        m2 = fminf(m2, fmaxf(m1, cm));
        chunk = cm < m1 ? c : chunk;
        m1 = fminf(m1, cm);
    }
    // The row's best column (relative to the segment) and exact second smallest.
    SLM_DEV void close(uint32_t &j, float &second) {
        uint32_t k1 = 0;
        float lo[8], hi[8];
#pragma unroll
        for (int k = 15; k >= 0; --k) k1 = cls[k] == m1 ? k : k1;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            lo[k] = fminf(cls[k], cls[k + 8]);
            hi[k] = fmaxf(cls[k], cls[k + 8]);
        }
#pragma unroll
        for (int n = 4; n; n >>= 1)
#pragma unroll
            for (int k = 0; k < n; ++k) {
                hi[k] = min3f(hi[k], hi[k + n], fmaxf(lo[k], lo[k + n]));
                lo[k] = fminf(lo[k], lo[k + n]);
            }
        j = chunk * 16 + k1;
        second = fminf(m2, hi[0]);
    }
};

// bar.sync of `n` threads that also returns the AND of ok over them.
SLM_DEV bool bar_and(int id, int n, bool ok) {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.u32 p, %3, 0;\n"
        "bar.red.and.pred q, %1, %2, p;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(r)
        : "r"(id), "r"(n), "r"((uint32_t)ok)
        : "memory");
    return r != 0;
}

// Instruction descriptor: bf16 inputs, f32 accumulate, K-major A and B, M = 128.
__host__ __device__ constexpr uint32_t top_idesc(uint32_t n, bool negate_b) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((negate_b ? 1u : 0u) << 14) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// Tier 1 (the BF16 rescue of an FP8 plan) works on the rescued pairs only.
SLM_DEV bool top_item_off(const SlArgs &g, const TopItem &it) {
    return g.tier && !sl_pair_on(g, g.spairs[it.pair]);
}

template <bool DUMP>
__global__ void __maxnreg__(96) sl_top2_kernel(SlArgs g) {
    grid_wait();
    extern __shared__ uint8_t top_smem_raw[];
    const uint32_t pad = (1024u - (smem_u32(top_smem_raw) & 1023u)) & 1023u;
    TopSmem &S = *reinterpret_cast<TopSmem *>(top_smem_raw + pad);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *err = g.ctl + 1;
    volatile uint32_t *abort_flag = &S.abort_flag;

    if (threadIdx.x == 0) {
        mbar_init(&S.a_full, 1);
        mbar_init(&S.a_empty, 1);
        for (int s = 0; s < kTopStages; ++s) {
            mbar_init(&S.b_full[s], 1);
            mbar_init(&S.b_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&S.t_full[b], 1);
            mbar_init(&S.t_empty[b], kTopEpWarps);
        }
        S.abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(&S.tmem_base, 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    const uint32_t it0 = g.tstart[blockIdx.x], it1 = g.tstart[blockIdx.x + 1];

    if (warp == 0) {
        // ---------------------------------------------------------- producer
        if (lane == 0) {
            uint32_t st = 0, sph = 0, loads = 0, issued = 0, cur = 0xffffffffu;
            bool ok = true;
            for (uint32_t it = it0; it < it1 && ok; ++it) {
                const TopItem item = g.titems[it];
                if (top_item_off(g, item)) continue;
                if (item.a_tile != cur) {
                    if (loads && !(ok = sl_wait(&S.a_empty, (loads - 1) & 1, abort_flag, err))) break;
                    cur = item.a_tile;
                    ++loads;
                    mbar_arrive_expect_tx(&S.a_full, item.nat * kBf16TileStride);
                    for (uint32_t a = 0; a < item.nat; ++a)
                        bulk_g2s(S.A[a], g.optiles + (size_t)(item.a_tile + a) * kBf16TileStride, kBf16TileStride,
                                 &S.a_full);
                }
                for (uint32_t t = 0; t < item.nt; t += 2) {
                    if (!(ok = sl_wait(&S.b_empty[st], sph ^ 1, abort_flag, err))) break;
                    const uint32_t n = min(2u, item.nt - t);
                    mbar_arrive_expect_tx(&S.b_full[st], n * kBf16TileStride);
                    ++issued;
                    for (uint32_t u = 0; u < n; ++u) {
                        const uint8_t *src = g.optiles + (size_t)(item.b_tile + t + u) * kBf16TileStride;
                        bulk_g2s(S.B[st] + u * kKb, src, kKb, &S.b_full[st]);
                        bulk_g2s(S.B[st] + (2 + u) * kKb, src + kKb, kKb, &S.b_full[st]);
                        bulk_g2s(S.B[st] + kStageExt + u * kBf16ExtBytes, src + 2 * kKb, kBf16ExtBytes, &S.b_full[st]);
                    }
                    if (++st == kTopStages) st = 0, sph ^= 1;
                }
            }
            drain_loads(S.b_full, kTopStages, issued);
            drain_loads(&S.a_full, 1, loads);
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issue
        // descriptors of fixed shared-memory addresses; a tile, stage or K step
        // adds its byte offset / 16 (all addresses lie below 256 KiB: no carry).
        // The norm extension of a row is one 16-byte core matrix row per operand
        // role; leading offset 0 reads it twice along K, and it holds |v|^2 / 4.
        constexpr uint32_t kTile16 = kBf16TileStride >> 4, kStage16 = kStageBytes >> 4;
        const uint64_t ad0 = umma_desc(smem_u32(S.A[0])), bd0 = umma_desc(smem_u32(S.B[0]));
        const uint64_t ax0 = umma_desc_plain(smem_u32(S.A[0]) + 2 * kKb, 0, 256);
        const uint64_t bx0 = umma_desc_plain(smem_u32(S.B[0]) + kStageExt + 128, 0, 256);
        uint32_t st = 0, sph = 0, tb = 0, tph = 0, loads = 0, cur = 0xffffffffu;
        bool ok = true;
        TopItem next = it0 < it1 ? g.titems[it0] : TopItem{};
        for (uint32_t it = it0; it < it1 && ok; ++it) {
            const TopItem item = next;
            if (it + 1 < it1) next = g.titems[it + 1];
            if (top_item_off(g, item)) continue;
            if (item.a_tile != cur) {
                if (loads && lane == 0) mma_commit(&S.a_empty);
                if (!(ok = sl_wait(&S.a_full, loads & 1, abort_flag, err))) break;
                cur = item.a_tile;
                ++loads;
            }
            for (uint32_t t = 0; t < item.nt && ok; t += 2) {
                if (!(ok = sl_wait(&S.b_full[st], sph, abort_flag, err))) break;
                // the pair's columns only, to the next 16 (1.73 -> 1.72 ms on the zone:
                // tiles of zeros cost time, but little power, and power sets the clock)
                const uint32_t n = (min(item.ncols - t * kTile, 256u) + 15) & ~15u;
                const uint32_t idesc = top_idesc(n, false), idesc_neg = top_idesc(n, true);
#pragma unroll
                for (uint32_t a = 0; a < 2; ++a) {
                    if (a >= item.nat) break;
                    if (!(ok = sl_wait(&S.t_empty[tb], tph ^ 1, abort_flag, err))) break;
                    tc_fence_after();
                    if (lane == 0) {
                        const uint32_t d = tmem + tb * 256;
                        const uint64_t ad = ad0 + (uint64_t)(a * kTile16), bd = bd0 + (uint64_t)(st * kStage16);
#pragma unroll
                        for (int k = 0; k < 8; ++k)  // K = 16 bf16 = 32 bytes per step; -a.b
                            mma_f16(d, ad + (k >> 2) * (kKb >> 4) + (k & 3) * 2,
                                    bd + (k >> 2) * (2 * kKb >> 4) + (k & 3) * 2, idesc_neg, k > 0);
                        // + (|a|^2 + |b|^2) / 2
                        mma_f16(d, ax0 + (uint64_t)(a * kTile16), bx0 + (uint64_t)(st * kStage16), idesc, true);
                        mma_commit(&S.t_full[tb]);
                    }
                    __syncwarp();
                    tb ^= 1;
                    if (tb == 0) tph ^= 1;
                }
                if (lane == 0) mma_commit(&S.b_empty[st]);
                __syncwarp();
                if (++st == kTopStages) st = 0, sph ^= 1;
            }
        }
    } else {
        // ---------------------------------------------------------- epilogue
        const int q = warp & 3, cg = (warp - 2) >> 2;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        const int row = q * 32 + lane;
        uint32_t tb = 0, tph = 0;
        bool ok = true;
        for (uint32_t it = it0; it < it1 && ok; ++it) {
            const TopItem item = g.titems[it];
            if (top_item_off(g, item)) continue;
            RowTop s[2];
            s[0].reset();
            s[1].reset();
            for (uint32_t t = 0; t < item.nt && ok; t += 2) {
                // chunks of this stage holding columns of the pair (the rest are padding)
                const uint32_t left = item.ncols - t * kTile;
                const uint32_t nch = (min(left, 256u) + 15) / 16, c0 = t * (kTile / 16);
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    if (a >= (int)item.nat) break;
                    if (!(ok = sl_wait(&S.t_full[tb], tph, abort_flag, err))) break;
                    tc_fence_after();
                    const uint32_t tcol = tmem + lane_addr + tb * 256;
                    if constexpr (DUMP) {
                        if (item.pair == 0 && !item.dir) {
                            const PairMeta pm = g.pairs[0];
                            const uint32_t i = (item.a_tile + a) * kTile - pm.a_row0 + row;
                            for (uint32_t c = cg; c < nch; c += 4) {
                                uint32_t v[16];
                                tmem_ld16(tcol + c * 16, v);
                                tmem_wait_ld16(v);
                                for (int k = 0; k < 16; ++k) {
                                    const uint32_t j = item.j0 + (c0 + c) * 16 + k;
                                    if (i < pm.na && j < pm.nb)
                                        g.dump[(size_t)i * pm.nb + j] = 2.f * __uint_as_float(v[k]);
                                }
                            }
                        }
                    }
                    uint32_t c = cg;
#pragma unroll 1
                    for (; c + 4 < nch; c += 8) {
                        uint32_t v0[16], v1[16], n0, n1;
                        tmem_ld16_min(tcol + c * 16, v0, n0);
                        tmem_ld16_min(tcol + c * 16 + 64, v1, n1);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(n0), "+r"(n1)::"memory");
                        tmem_tie16(v0);
                        tmem_tie16(v1);
#pragma unroll
                        for (int k = 0; k < 16; ++k)
                            s[a].cls[k] = min3f(s[a].cls[k], __uint_as_float(v0[k]), __uint_as_float(v1[k]));
                        s[a].add_min(__uint_as_float(n0), c0 + c);
                        s[a].add_min(__uint_as_float(n1), c0 + c + 4);
                    }
                    if (c < nch) {
                        uint32_t v0[16], n0;
                        tmem_ld16_min(tcol + c * 16, v0, n0);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(n0)::"memory");
                        tmem_tie16(v0);
#pragma unroll
                        for (int k = 0; k < 16; ++k) s[a].cls[k] = fminf(s[a].cls[k], __uint_as_float(v0[k]));
                        s[a].add_min(__uint_as_float(n0), c0 + c);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&S.t_empty[tb]);
                    tb ^= 1;
                    if (tb == 0) tph ^= 1;
                }
            }
            // the four column groups of a lane quarter merge: group a keeps a
            // tile a's rows, the others hand theirs over (a barrier of the
            // quarter's 128 threads before the buffer is written, one after).
            // The first barrier also makes a timed-out wait the whole quarter's,
            // so that no warp waits at a later item for one that has left.
            float m1[2], m2[2];
            uint32_t j[2];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                s[a].close(j[a], m2[a]);
                m1[a] = s[a].m1;
            }
            ok = bar_and(q + 1, 128, ok);
#pragma unroll
            for (int a = 0; a < 2; ++a)
                if (cg != a) {
                    const int slot = cg < a ? cg : cg - 1;
                    S.mm[a][slot][row] = make_float2(m1[a], m2[a]);
                    S.mj[a][slot][row] = j[a];
                }
            asm volatile("bar.sync %0, 128;" ::"r"(q + 1) : "memory");
#pragma unroll
            for (int a = 0; a < 2; ++a)
                if (cg == a && a < (int)item.nat && ok) {
                    float b1 = m1[a], b2 = m2[a];
                    uint32_t bj = j[a];
#pragma unroll
                    for (int o = 0; o < 3; ++o) {
                        const float2 v = S.mm[a][o][row];
                        top2_merge(b1, b2, bj, v.x, v.y, S.mj[a][o][row]);
                    }
                    const size_t out = ((size_t)item.part << g.tshift) + a * kTile + row;
                    g.topmm[out] = make_float2(2.f * b1, 2.f * b2);  // d~ from d~ / 2
                    g.topj[out] = item.j0 + bj;
                }
        }
    }
    // Everyone done: no MMA in flight (the epilogue consumed every commit).
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------- decisions

// A row's two smallest estimates and nearest column: its segments' results
// merged (one segment but where a CTA's share of the work ended inside its
// columns). blk0: the side's first block.
SLM_DEV void row_top2(const SlArgs &g, uint32_t blk0, uint32_t i, float &m1, float &m2, uint32_t &j) {
    const uint2 b = g.tblk[blk0 + (i >> g.tshift)];  // {first part, parts}
    const size_t r = ((size_t)b.x << g.tshift) + (i & ((1u << g.tshift) - 1));
    const float2 v = g.topmm[r];
    m1 = v.x;
    m2 = v.y;
    j = g.topj[r];
    for (uint32_t s = 1; s < b.y; ++s) {
        const size_t o = r + ((size_t)s << g.tshift);
        const float2 w = g.topmm[o];
        top2_merge(m1, m2, j, w.x, w.y, g.topj[o]);
    }
}

// The cross-check of row i, whose exact distance to its nearest column j is at
// least dlow, from the column's two smallest estimates c1 (at row i1) and c2:
// the column's nearest row is certain when every other row's estimate is more
// than 2 eps above its best one; row i is certainly not it when dlow lies above
// the largest distance the best row may have. Anything else is queued for an
// exact column scan.
SLM_DEV uint32_t mutual_decision(const SlArgs &g, uint32_t p, float eps, uint32_t i, uint32_t j, float dlow, float c1,
                                 float c2, uint32_t i1) {
    if (__fsub_rd(c2, c1) > 2.f * eps) return i1 == i ? j : kDecNone;
    if (dlow > __fadd_ru(c1, eps)) return kDecNone;
    push_scan(g, p, 1, i, j);
    return kDecPending;
}
SLM_DEV uint32_t mutual_from_top2(const SlArgs &g, uint32_t p, const SlPair &sp, uint32_t i, uint32_t j, float dlow) {
    float c1, c2;
    uint32_t i1;
    row_top2(g, sp.tblk_b, j, c1, c2, i1);
    return mutual_decision(g, p, sp.eps, i, j, dlow, c1, c2, i1);
}

// Row i of pair p joins the undecided rows of its b view; whoever starts a new
// run of 16 or 128 there registers that run as a group for the resolve kernels.
SLM_DEV void list_undecided(const SlArgs &g, const SlPair &sp, uint32_t p, uint32_t i) {
    const uint32_t k = atomicAdd(&g.ucnt[sp.ubucket], 1u);
    g.ulist[sp.ubase + k] = make_uint2(p, i);
    if (k % kGroupRows == 0)
        g.ugroups[atomicAdd(&g.ctl[kCtlGroups], 1u)] = make_uint4(sp.ubase + k, sp.ubucket, k, 0u);
    if (k % kTileRows == 0)
        g.utiles[atomicAdd(&g.ctl[kCtlTiles], 1u)] = make_uint4(sp.ubase + k, sp.ubucket, k, 0u);
}

// A row whose ratio test the estimates leave open, its nearest column j certain
// and e1 its exact distance: only the second best's error remains. Returns
// false when that still leaves it open.
SLM_DEV bool settle_with_d1(const SlArgs &g, const SlPair &sp, uint32_t p, uint32_t i, uint32_t j, float e1, float m2) {
    const bool fails = e1 >= __fmul_ru(__fmul_ru(g.ratio2, __fadd_ru(m2, sp.eps)), kUp);
    const bool passes = e1 < __fmul_rd(__fmul_rd(g.ratio2, __fsub_rd(m2, sp.eps)), kDown);
    if (!fails && !passes) return false;
    g.rowdec[sp.rbase + i] = fails ? kDecNone : g.mutual ? mutual_from_top2(g, p, sp, i, j, e1) : j;
    return true;
}

// CTA per pair and kDecideThreads x R rows of a, R rows a thread: the outcome
// the bounds certify. A row whose nearest column is certain but whose ratio
// test is not gets its exact d1 (settle_with_d1): 3 of 5 such rows, for 1 KB
// read each, of those that sl_resolve_kernel would read a whole view for.
// A row is a chain of dependent loads (block, result, the column's block and
// result). R = 4 keeps four of them going in a thread (71 -> 54 us for the
// 4.2 M rows of a zone) and lists the open rows for sl_nearest_kernel, 20 us
// there. Batches too small to fill the GPU that way run R = 1 and take the
// exact d1 in the CTA that finds the row (one 8192 pair: 13 us against 10 and
// 13 in a kernel of its own).
constexpr uint32_t kDecideThreads = 256;
template <int R>
__global__ void __launch_bounds__(kDecideThreads) sl_decide_kernel(SlArgs g, uint32_t block0) {
    grid_wait();
    grid_go();
    const uint32_t p = blockIdx.x, row0 = (block0 + blockIdx.y) * (kDecideThreads * R);
    const PairMeta pm = g.pairs[p];
    if (row0 >= pm.na) return;  // block-uniform, as below
    const SlPair sp = g.spairs[p];
    if (!sl_pair_on(g, sp)) return;
    __shared__ uint4 found[R == 1 ? kDecideThreads : 1];  // R = 1: this CTA's open rows
    __shared__ uint32_t n_found, n_settled;
    if (R == 1 && threadIdx.x == 0) n_found = n_settled = 0;
    if (R == 1) __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const float eps = sp.eps;
    uint32_t j[R], dec[R];
    float m1[R], m2[R];
    bool match[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t i = row0 + r * kDecideThreads + threadIdx.x;
        m1[r] = m2[r] = __int_as_float(0x7f800000);
        j[r] = 0;
        if (i < pm.na && pm.nb) row_top2(g, sp.tblk_a, i, m1[r], m2[r], j[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        // fewer than two columns: the exact second best is infinite (matching.rs:205)
        const bool some = m2[r] < __int_as_float(0x7f800000) && !certain_no_match(m1[r], m2[r], eps, g.ratio2);
        const bool unique = __fsub_rd(m2[r], m1[r]) > 2.f * eps;  // every other column is farther
        match[r] = some && unique && certain_ratio_pass(m1[r], m2[r], eps, g.ratio2);
        dec[r] = match[r] ? j[r] : some ? kDecPending : kDecNone;
        const bool open = some && !match[r];
        const uint32_t m = __ballot_sync(0xffffffffu, open);
        if (m) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(R == 1 ? &n_found : &g.ctl[kCtlOpen], (uint32_t)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (open)
                (R == 1 ? found : g.olist)[base + __popc(m & ((1u << lane) - 1))] =
                    make_uint4(p, row0 + r * kDecideThreads + threadIdx.x, unique ? j[r] : kDecNone,
                               __float_as_uint(m2[r]));
        }
    }
    if (g.mutual) {
        float c1[R], c2[R];
        uint32_t i1[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (match[r]) row_top2(g, sp.tblk_b, j[r], c1[r], c2[r], i1[r]);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (match[r])
                dec[r] = mutual_decision(g, p, eps, row0 + r * kDecideThreads + threadIdx.x, j[r],
                                         __fsub_rd(m1[r], eps), c1[r], c2[r], i1[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t i = row0 + r * kDecideThreads + threadIdx.x;
        if (i < pm.na) g.rowdec[sp.rbase + i] = dec[r];
    }
    if constexpr (R == 1) {
        __syncthreads();  // the open rows are listed, and their decisions written as pending
        for (uint32_t s0 = (threadIdx.x / 32) * 4; s0 < n_found; s0 += kDecideThreads / 8) {  // warp-uniform
            const uint32_t s = s0 + (lane >> 3);
            const uint4 o = found[min(s, n_found - 1)];
            const bool exact = o.z != kDecNone;
            const float e1 = dist8(g.raw + (size_t)(pm.a_raw0 + o.y) * kDesc,
                                   g.raw + (size_t)(pm.b_raw0 + (exact ? o.z : 0)) * kDesc);
            if (s < n_found && (lane & 7) == 0) {
                if (exact && settle_with_d1(g, sp, p, o.y, o.z, e1, __uint_as_float(o.w)))
                    atomicAdd(&n_settled, 1u);
                else
                    list_undecided(g, sp, p, o.y);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && n_settled) atomicAdd(&g.ctl[kCtlRescored], n_settled);
    }
}

// The open rows of a large batch, two lanes each.
__global__ void __launch_bounds__(256) sl_nearest_kernel(SlArgs g) {
    grid_wait();
    grid_go();
    const uint32_t lane = threadIdx.x & 31, n = g.ctl[kCtlOpen];
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    uint32_t settled = 0;
    for (uint32_t s0 = gw * 16; s0 < n; s0 += nw * 16) {  // warp-uniform
        const uint32_t s = s0 + (lane >> 1);
        const uint4 o = g.olist[min(s, n - 1)];
        const PairMeta pm = g.pairs[o.x];
        const SlPair sp = g.spairs[o.x];
        const bool exact = o.z != kDecNone;
        const float e1 = dist2(g.raw + (size_t)(pm.a_raw0 + o.y) * kDesc,
                               g.raw + (size_t)(pm.b_raw0 + (exact ? o.z : 0)) * kDesc);
        if (s < n && (lane & 1) == 0) {
            if (exact && settle_with_d1(g, sp, o.x, o.y, o.z, e1, __uint_as_float(o.w)))
                ++settled;
            else
                list_undecided(g, sp, o.x, o.y);
        }
    }
    settled = __reduce_add_sync(0xffffffffu, settled);
    if (lane == 0 && settled) atomicAdd(&g.ctl[kCtlRescored], settled);
}

// --------------------------------------------------------------- resolve

// Undecided rows: the estimates against every column of their b view once more, the
// columns within the window m2 + 2 eps, the exact distances of those, and the
// reference's row rule (matching.rs:182-187, 204-206). Rows are grouped by b view over
// all pairs, since reading the view is the cost: in tens of us by sl_resolve_kernel
// where they are few, by sl_resolve_tile_kernel in groups of 128 where they are many,
// whichever the estimate of the two finds shorter (both are launched, one returns).
// With groups of 16 alone a 32768 x 32768 pair with every row undecided took 4.0 ms, or
// 7.7 with shortlists of 32 columns, whose overflows are scanned; with groups of 128
// alone 30 pairs of 500 to 4000 rows took 134 us instead of 126, and one pair of 8192
// rows 172 instead of 161, from the larger CTAs' start.
// us, measured: groups of 16 take about 18 and 1.3 a tile of a CTA of their cluster, in
// rounds of the launch's clusters; groups of 128 about 15 and 0.6 a tile, in rounds of CTAs,
// and 20 to start.
SLM_DEV bool resolve_by_tiles(const SlArgs &g) {
    const float few = ceilf((float)g.ctl[kCtlGroups] * (float)g.few_cluster / (float)g.few_ctas) *
                      (18.f + 1.3f * g.mean_tiles / (float)g.few_cluster);
    const float many = ceilf((float)g.ctl[kCtlTiles] / (float)g.res_ctas) * (15.f + 0.6f * g.mean_tiles);
    return few > 20.f + 1.2f * many;
}

// A row with more columns in its window than a shortlist holds is scanned exactly; a
// pair with more than 1/8 such rows goes to the exact kernel.
SLM_DEV void scan_instead(const SlArgs &g, uint32_t p, const PairMeta &pm, uint32_t i) {
    push_scan(g, p, 0, i, 0);
    const uint32_t was = atomicAdd(&g.pairctl[4 * (size_t)p + kPcOver], 1u);
    if (was * 8 <= pm.na && (was + 1) * 8 > pm.na) {
        g.spairs[p].routed = 1;
        atomicAdd(&g.ctl[kCtlRouteMarks], 1u);
    }
}

// A row's decision from its exact two smallest distances.
SLM_DEV void decide_exact(const SlArgs &g, uint32_t p, const SlPair &sp, uint32_t i, float e1, float e2, uint32_t ej) {
    uint32_t dec = kDecNone;
    if (ej != 0xffffffffu && e2 < __int_as_float(0x7f800000) && !(e1 >= __fmul_rn(g.ratio2, e2)))
        dec = g.mutual ? mutual_from_top2(g, p, sp, i, ej, e1) : ej;
    g.rowdec[sp.rbase + i] = dec;
}

SLM_DEV void merge_exact(float &e1, float &e2, uint32_t &ej, float o1, float o2, uint32_t oj) {
    e2 = fminf(fminf(e2, o2), fmaxf(e1, o1));
    if (o1 < e1 || (o1 == e1 && oj < ej)) {
        e1 = o1;
        ej = oj;
    }
}

SLM_DEV void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The 16-byte chunk c (0..15) of store row r of the BF16 operand image.
SLM_DEV uint4 op_chunk(const SlArgs &g, uint32_t r, uint32_t c) {
    const uint8_t *t = g.optiles + (size_t)(r / kTile) * kBf16TileStride + (c >> 3) * kKb + (r % kTile) * 128;
    return *reinterpret_cast<const uint4 *>(t + (((c & 7) ^ (r & 7)) * 16));
}

// Few undecided rows: one cluster per group of 16 of one b view. The group's rows
// lie scattered over views, and 16 are a warp-level tile exactly: m16n8k16 with both
// operands straight from the operand image, without staging. The sum over k may run in
// any order, so lane t of four takes the 16-byte chunks 4 q + t of its row, on
// both sides, and each chunk is the operand words of two steps.
// Reading the b view (256 bytes a column) is the cost, so rows are grouped by b
// view over all pairs, and the cluster's CTAs share a group's columns: a large
// view is not one CTA's chain of loads. The candidates meet in CTA 0's shared
// memory, and the exact distances are spread over the cluster's warps again.
// A row with more columns in the window than g.cand_cap is scanned exactly
// instead; a pair with more than 1/8 such rows goes to the exact kernel.
__global__ void __launch_bounds__(256) sl_resolve_kernel(SlArgs g) {
    grid_wait();
    grid_go();
    if (resolve_by_tiles(g)) return;
    constexpr uint32_t kCap = kResolveCols;
    __shared__ uint32_t cand_s[kGroupRows][kCap];
    __shared__ float cval_s[kGroupRows][kCap];
    __shared__ uint32_t cnt_s[kGroupRows];
    __shared__ uint2 rows[kGroupRows];
    __shared__ uint32_t arow[kGroupRows];
    __shared__ float win[kGroupRows], nrm[kGroupRows];
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const uint32_t rank = cl.block_rank(), ncta = cl.num_blocks();
    uint32_t (*cand)[kCap] = cl.map_shared_rank(cand_s, 0);
    float (*cval)[kCap] = cl.map_shared_rank(cval_s, 0);
    uint32_t *cnt = cl.map_shared_rank(cnt_s, 0);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t gr = lane >> 2, t = lane & 3;
    const uint32_t gwarp = rank * (blockDim.x / 32) + warp, nwarp = ncta * (blockDim.x / 32);
    const float kInf = __int_as_float(0x7f800000);
    const uint32_t ng = g.ctl[kCtlGroups];
    uint32_t w_rows = 0;
    float w_err = 0.f;
    for (uint32_t e = blockIdx.x / ncta; e < ng; e += gridDim.x / ncta) {
        const uint4 ug = g.ugroups[e];
        const uint32_t n = min(kGroupRows, g.ucnt[ug.y] - ug.z);
        const PairMeta pb = g.pairs[g.ulist[ug.x].x];  // every pair of the group has this b view
        if (tid < kGroupRows) {
            // rows past the list's end repeat its first row and admit nothing
            const uint2 r = g.ulist[ug.x + (tid < n ? tid : 0)];
            const SlPair sp = g.spairs[r.x];
            float m1, m2;
            uint32_t j;
            row_top2(g, sp.tblk_a, r.y, m1, m2, j);
            rows[tid] = r;
            arow[tid] = g.pairs[r.x].a_row0 + r.y;
            cnt_s[tid] = 0;
            win[tid] = tid < n ? window_up(m2, sp.eps) : -kInf;
            nrm[tid] = g.norms[arow[tid]];
        }
        cl.sync();
        uint32_t A[2][16];  // rows gr and gr + 8: word w of chunk q is A[.][4 q + w]
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = op_chunk(g, arow[gr + 8 * h], 4 * q + t);
                A[h][4 * q] = v.x, A[h][4 * q + 1] = v.y, A[h][4 * q + 2] = v.z, A[h][4 * q + 3] = v.w;
            }
        const float na0 = nrm[gr], na1 = nrm[gr + 8], w0 = win[gr], w1 = win[gr + 8];
        const uint32_t n8 = (pb.nb + 7) / 8;  // columns past nb have a NaN norm: never admitted
        for (uint32_t c8 = gwarp; c8 < n8; c8 += 2 * nwarp) {
            uint4 B[2][4];
            const bool two = c8 + nwarp < n8;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t r = pb.b_row0 + (c8 + (u && two ? nwarp : 0)) * 8 + gr;
#pragma unroll
                for (int q = 0; q < 4; ++q) B[u][q] = op_chunk(g, r, 4 * q + t);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (u && !two) break;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    mma_16816(acc, A[0][4 * q], A[1][4 * q], A[0][4 * q + 1], A[1][4 * q + 1], B[u][q].x, B[u][q].y);
                    mma_16816(acc, A[0][4 * q + 2], A[1][4 * q + 2], A[0][4 * q + 3], A[1][4 * q + 3], B[u][q].z,
                              B[u][q].w);
                }
                const uint32_t j = (c8 + nwarp * u) * 8 + 2 * t;
                const float2 nb = *reinterpret_cast<const float2 *>(g.norms + pb.b_row0 + j);
                const float d[4] = {fmaf(-2.f, acc[0], na0 + nb.x), fmaf(-2.f, acc[1], na0 + nb.y),
                                    fmaf(-2.f, acc[2], na1 + nb.x), fmaf(-2.f, acc[3], na1 + nb.y)};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (d[k] <= (k < 2 ? w0 : w1)) {
                        const uint32_t r = gr + (k < 2 ? 0 : 8);
                        const uint32_t s = atomicAdd(&cnt[r], 1u);
                        if (s < g.cand_cap) {
                            cand[r][s] = j + (k & 1);
                            cval[r][s] = d[k];
                        }
                    }
            }
        }
        cl.sync();
        // exact distances, 2 lanes a column: a warp per row where the cluster has
        // 16 warps, else 8 lanes per row, four rows of a warp side by side
        const uint32_t width = nwarp >= kGroupRows ? 32 : 8, sub = lane & (width - 1);
        const uint32_t per = 32 / width, cols = width / 2;
        for (uint32_t r0 = gwarp * per; r0 < n; r0 += nwarp * per) {  // warp-uniform
            const uint32_t r = min(r0 + lane / width, n - 1);
            const bool have = r0 + lane / width < n;
            const uint32_t p = rows[r].x, i = rows[r].y, m = cnt[r];
            const PairMeta pm = g.pairs[p];
            const SlPair sp = g.spairs[p];
            const float *a = g.raw + (size_t)(pm.a_raw0 + i) * kDesc;
            const float *B = g.raw + (size_t)pm.b_raw0 * kDesc;
            const bool over = m > g.cand_cap;
            const uint32_t mine_n = have && !over ? m : 0;
            const uint32_t most = __reduce_max_sync(0xffffffffu, mine_n);
            float e1 = kInf, e2 = kInf;
            uint32_t ej = 0xffffffffu;
            for (uint32_t s = 0; s < most; s += cols) {
                const uint32_t mine = s + (sub >> 1);
                const uint32_t j = mine < mine_n ? cand[r][mine] : 0;
                const float d = dist2(a, B + (size_t)j * kDesc);
                if (mine < mine_n) {
                    w_err = fmaxf(w_err, fabsf(d - cval[r][mine]));
                    if (d < e1 || (d == e1 && j < ej)) {
                        e2 = e1;
                        e1 = d;
                        ej = j;
                    } else if (d < e2) {
                        e2 = d;
                    }
                }
            }
            // over the row's lane pairs (no column occurs twice)
            for (uint32_t o = 2; o < width; o <<= 1) {
                const float o1 = __shfl_xor_sync(0xffffffffu, e1, o), o2 = __shfl_xor_sync(0xffffffffu, e2, o);
                const uint32_t oj = __shfl_xor_sync(0xffffffffu, ej, o);
                e2 = fminf(fminf(e2, o2), fmaxf(e1, o1));
                if (o1 < e1 || (o1 == e1 && oj < ej)) {
                    e1 = o1;
                    ej = oj;
                }
            }
            if (have && sub == 0) {
                if (over) {
                    scan_instead(g, p, pm, i);
                } else {
                    ++w_rows;
                    decide_exact(g, p, sp, i, e1, e2, ej);
                }
            }
        }
        cl.sync();  // CTA 0's lists are free, and no CTA leaves while they are read
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) w_err = fmaxf(w_err, __shfl_xor_sync(0xffffffffu, w_err, o));
    w_rows = __reduce_add_sync(0xffffffffu, w_rows);
    if (lane == 0 && w_rows) {
        atomicAdd(&g.ctl[kCtlRescored], w_rows);
        atomicMax(&g.ctl[kCtlMaxErr], __float_as_uint(w_err));  // non-negative: bits order as values
    }
}

constexpr uint32_t kResVals = 15;         // of a row's shortlist, with their estimates (for the largest error seen)
constexpr uint32_t kResRunTiles = 512;    // column tiles between two looks at the lists: 16 bits a column
struct ResSmem {
    uint8_t A[kBf16TileStride];
    uint8_t B[kTopStages][kStageBytes];
    uint16_t cand[kTileRows][kResolveCols];
    float cval[kTileRows][kResVals];
    float4 part[kTileRows];  // a row's two smallest exact distances, the column of the first, columns in the window
    uint2 rows[kTileRows];
    float thr[kTileRows];
    uint32_t cnt[kTileRows];
    uint64_t a_full;
    uint64_t b_full[kTopStages];
    uint64_t t_full[kTopStages], t_empty[kTopStages];  // t_full: also the b tiles are free again
    uint32_t tmem_base;
    uint32_t abort_flag;
};
constexpr size_t kResSmemBytes = sizeof(ResSmem) + 1024;  // slack for 1024-byte alignment
static_assert(kResSmemBytes <= 232448, "shared memory of one CTA");
static_assert(kTileRows == kTile && kTopStages == 2, "a group is one a tile, a stage's accumulator half of TMEM");

SLM_DEV void epilogue_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// Many undecided rows: one CTA per group of up to 128 of one b view. The epilogue's
// warps gather the rows, which lie scattered over views, from the operand image into one
// a tile, and the group is then a tile of the pass: sl_top2_kernel's roles, M = 128, N =
// 256. What is within a row's window is listed in shared memory, its exact distances
// taken once the view (or 65536 columns of it) is through. 0.55 us a tile of 128 columns,
// bound by the MMAs (0.36 in the pass, whose b tiles serve two a tiles); with many hits,
// which a warp appends by the chunk, up to 0.9. (N = 128: 0.95. A cluster's CTAs sharing
// the view's tiles and one list: 2.6 us for a tile of 12 hits.)
__global__ void __maxnreg__(96) sl_resolve_tile_kernel(SlArgs g) {
    grid_wait();
    grid_go();
    if (!resolve_by_tiles(g)) return;
    extern __shared__ uint8_t res_smem_raw[];
    const uint32_t pad = (1024u - (smem_u32(res_smem_raw) & 1023u)) & 1023u;
    ResSmem &S = *reinterpret_cast<ResSmem *>(res_smem_raw + pad);
    const uint32_t ng = g.ctl[kCtlTiles];
    if (blockIdx.x >= ng) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *err = g.ctl + 1;
    volatile uint32_t *abort_flag = &S.abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(&S.a_full, kTopEpWarps);
        for (int s = 0; s < kTopStages; ++s) {
            mbar_init(&S.b_full[s], 1);
            mbar_init(&S.t_full[s], 1);
            mbar_init(&S.t_empty[s], kTopEpWarps);
        }
        S.abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(&S.tmem_base, 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    const float kInf = __int_as_float(0x7f800000);
    uint32_t st = 0, sph = 0, iter = 0;  // stage and its phase; groups
    uint32_t issued = 0;                 // stages loaded
    uint32_t w_rows = 0;
    float w_err = 0.f;
    // (after a wait that gave up every role still goes through its groups, without waiting)
    for (uint32_t e = blockIdx.x; e < ng; e += gridDim.x, ++iter) {
        const uint4 ug = g.utiles[e];
        const PairMeta pb = g.pairs[g.ulist[ug.x].x];  // every pair of the group has this b view
        const uint32_t n = min(kTileRows, g.ucnt[ug.y] - ug.z);
        const uint32_t nt = (pb.nb + kTile - 1) / kTile;
        // columns of the stage from tile t on, rounded up to the MMA's and the loads' 16
        const auto columns = [&](uint32_t t) { return (min(2u * kTile, pb.nb - t * kTile) + 15) & ~15u; };
        if (warp == 0) {
            // ------------------------------------------------------ producer
            for (uint32_t t = 0; t < nt; t += 2) {
                if (lane == 0 && !*abort_flag && sl_wait(&S.t_full[st], sph ^ 1, abort_flag, err)) {
                    const uint32_t m = min(2u, nt - t);
                    mbar_arrive_expect_tx(&S.b_full[st], m * kBf16TileStride);
                    ++issued;
                    for (uint32_t u = 0; u < m; ++u) {
                        const uint8_t *src = g.optiles + (size_t)(pb.b_row0 / kTile + t + u) * kBf16TileStride;
                        bulk_g2s(S.B[st] + u * kKb, src, kKb, &S.b_full[st]);
                        bulk_g2s(S.B[st] + (2 + u) * kKb, src + kKb, kKb, &S.b_full[st]);
                        bulk_g2s(S.B[st] + kStageExt + u * kBf16ExtBytes, src + 2 * kKb, kBf16ExtBytes, &S.b_full[st]);
                    }
                }
                __syncwarp();
                if (++st == kTopStages) st = 0, sph ^= 1;
            }
        } else if (warp == 1) {
            // ---------------------------------------------------- MMA issue (as sl_top2_kernel's)
            const uint64_t ad = umma_desc(smem_u32(S.A)), ax = umma_desc_plain(smem_u32(S.A) + 2 * kKb, 0, 256);
            const uint64_t bd0 = umma_desc(smem_u32(S.B[0])), bx0 = umma_desc_plain(smem_u32(S.B[0]) + kStageExt + 128, 0, 256);
            bool ok = !*abort_flag && sl_wait(&S.a_full, iter & 1, abort_flag, err);
            for (uint32_t t = 0; t < nt && ok; t += 2) {
                ok = sl_wait(&S.b_full[st], sph, abort_flag, err) && sl_wait(&S.t_empty[st], sph ^ 1, abort_flag, err);
                if (!ok) break;
                tc_fence_after();
                if (lane == 0) {
                    const uint32_t cols = columns(t);
                    const uint32_t d = tmem + st * 256, idesc = top_idesc(cols, false), idesc_neg = top_idesc(cols, true);
                    const uint64_t stage = (uint64_t)(st * (kStageBytes >> 4));
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        mma_f16(d, ad + (k >> 2) * (kKb >> 4) + (k & 3) * 2,
                                bd0 + stage + (k >> 2) * (2 * kKb >> 4) + (k & 3) * 2, idesc_neg, k > 0);
                    mma_f16(d, ax, bx0 + stage, idesc, true);
                    mma_commit(&S.t_full[st]);
                }
                __syncwarp();
                if (++st == kTopStages) st = 0, sph ^= 1;
            }
            __syncwarp();
        } else {
            // ------------------------------------------------------ epilogue
            {  // four threads a row: its operand image (128 bytes of each K block, the norm extension)
                const uint32_t et = threadIdx.x - 64, row = et >> 2, part = et & 3;
                // rows past the list's end repeat its first row and admit nothing
                const uint2 r = g.ulist[ug.x + (row < n ? row : 0)];
                const uint32_t ar = g.pairs[r.x].a_row0 + r.y, rr = ar % kTile;
                const uint8_t *src = g.optiles + (size_t)(ar / kTile) * kBf16TileStride;
                uint4 v[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t c = part * 4 + k;
                    v[k] = *reinterpret_cast<const uint4 *>(src + (c >> 3) * kKb + rr * 128 + (((c & 7) ^ (rr & 7)) * 16));
                }
                epilogue_sync();  // the group before: its MMAs are done, its rows were read until here
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t c = part * 4 + k;
                    *reinterpret_cast<uint4 *>(S.A + (c >> 3) * kKb + row * 128 + (((c & 7) ^ (row & 7)) * 16)) = v[k];
                }
                if (part == 0) {
                    *reinterpret_cast<uint4 *>(S.A + 2 * kKb + (row >> 3) * 256 + (row & 7) * 16) =
                        *reinterpret_cast<const uint4 *>(src + 2 * kKb + (rr >> 3) * 256 + (rr & 7) * 16);
                } else if (part == 1) {
                    S.rows[row] = r;
                    S.cnt[row] = 0;
                    S.part[row] = make_float4(kInf, kInf, __uint_as_float(0xffffffffu), 0.f);
                } else if (part == 2) {
                    const SlPair sp = g.spairs[r.x];
                    float m1, m2;
                    uint32_t j;
                    row_top2(g, sp.tblk_a, r.y, m1, m2, j);
                    S.thr[row] = row < n ? 0.5f * window_up(m2, sp.eps) : -kInf;  // of d~ / 2
                }
                fence_proxy_async();  // the MMAs read what this thread wrote
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.a_full);
            }
            for (uint32_t run = 0; run < nt; run += kResRunTiles) {
                epilogue_sync();  // the lists are empty
                const int q = warp & 3, cg = (warp - 2) >> 2, row = q * 32 + lane;
                const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
                const float thr = S.thr[row];
                for (uint32_t t = run; t < min(run + kResRunTiles, nt); t += 2) {
                    if (*abort_flag || !sl_wait(&S.t_full[st], sph, abort_flag, err)) break;
                    tc_fence_after();
                    const uint32_t tcol = tmem + lane_addr + st * 256, nch = columns(t) / 16;
                    for (uint32_t c = cg; c < nch; c += 4) {
                        uint32_t v[16], mn;
                        tmem_ld16_min(tcol + c * 16, v, mn);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(mn)::"memory");
                        tmem_tie16(v);
                        if (__uint_as_float(mn) <= thr) {  // columns past nb have NaN estimates: never admitted
                            uint32_t hits = 0;
#pragma unroll
                            for (int k = 0; k < 16; ++k) hits |= __uint_as_float(v[k]) <= thr ? 1u << k : 0u;
                            // a lone hit's estimate is the chunk's minimum; of several, none is kept
                            const float val = (hits & (hits - 1)) ? __int_as_float(0x7fc00000) : 2.f * __uint_as_float(mn);
                            uint32_t s = atomicAdd(&S.cnt[row], (uint32_t)__popc(hits));
                            const uint32_t j = (t - run) * kTile + c * 16 - 1;
                            for (; hits; hits &= hits - 1, ++s) {
                                if (s < kResolveCols) S.cand[row][s] = (uint16_t)(j + __ffs(hits));
                                if (s < kResVals) S.cval[row][s] = val;
                            }
                        }
                        __syncwarp();
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&S.t_empty[st]);
                    if (++st == kTopStages) st = 0, sph ^= 1;
                }
                epilogue_sync();
                // exact distances of this CTA's columns, 2 lanes each: four rows of a warp side by
                // side, or all its lanes on one where there are as many warps
                const uint32_t width = n <= kTopEpWarps ? 32 : n <= 2 * kTopEpWarps ? 16 : 8, sub = lane & (width - 1);
                const uint32_t per = 32 / width, cols = width / 2;
                for (uint32_t r0 = (warp - 2) * per; r0 < n; r0 += kTopEpWarps * per) {  // warp-uniform
                    const uint32_t r = min(r0 + lane / width, n - 1), m = S.cnt[r];
                    const bool have = r0 + lane / width < n;
                    const PairMeta pm = g.pairs[S.rows[r].x];
                    const float *a = g.raw + (size_t)(pm.a_raw0 + S.rows[r].y) * kDesc;
                    const float *B = g.raw + (size_t)(pm.b_raw0 + (uint64_t)run * kTile) * kDesc;
                    const uint32_t mine_n = have && m <= g.cand_cap ? m : 0;
                    const uint32_t most = __reduce_max_sync(0xffffffffu, mine_n);
                    float e1 = kInf, e2 = kInf;
                    uint32_t ej = 0xffffffffu;
                    for (uint32_t s = 0; s < most; s += cols) {
                        const uint32_t mine = s + (sub >> 1);
                        const uint32_t j = mine < mine_n ? S.cand[r][mine] : 0;
                        const float d = dist2<8>(a, B + (size_t)j * kDesc);
                        if (mine < mine_n) {
                            if (mine < kResVals) w_err = fmaxf(w_err, fabsf(d - S.cval[r][mine]));
                            merge_exact(e1, e2, ej, d, kInf, run * kTile + j);
                        }
                    }
                    // over the row's lane pairs (no column occurs twice)
                    for (uint32_t o = 2; o < width; o <<= 1)
                        merge_exact(e1, e2, ej, __shfl_xor_sync(0xffffffffu, e1, o), __shfl_xor_sync(0xffffffffu, e2, o),
                                    __shfl_xor_sync(0xffffffffu, ej, o));
                    if (have && sub == 0) {
                        float4 &p = S.part[r];  // with the runs before
                        merge_exact(e1, e2, ej, p.x, p.y, __float_as_uint(p.z));
                        p = make_float4(e1, e2, __uint_as_float(ej), __uint_as_float(__float_as_uint(p.w) + m));
                        S.cnt[r] = 0;
                    }
                }
            }
            epilogue_sync();
            const uint32_t r = threadIdx.x - 64;  // a thread a row
            if (r < n) {
                const float4 v = S.part[r];
                const uint32_t p = S.rows[r].x, i = S.rows[r].y;
                if (__float_as_uint(v.w) > g.cand_cap) {
                    scan_instead(g, p, g.pairs[p], i);
                } else {
                    ++w_rows;
                    decide_exact(g, p, g.spairs[p], i, v.x, v.y, __float_as_uint(v.z));
                }
            }
            __syncwarp();
        }
    }
    if (warp == 0 && lane == 0) drain_loads(S.b_full, kTopStages, issued);
    __syncwarp();
    if (warp >= 2) {
#pragma unroll
        for (int o = 16; o; o >>= 1) w_err = fmaxf(w_err, __shfl_xor_sync(0xffffffffu, w_err, o));
        w_rows = __reduce_add_sync(0xffffffffu, w_rows);
        if (lane == 0) {
            if (w_rows) atomicAdd(&g.ctl[kCtlRescored], w_rows);
            if (w_err > 0.f) atomicMax(&g.ctl[kCtlMaxErr], __float_as_uint(w_err));  // non-negative: bits order as values
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace

cudaError_t init_top2_kernels() {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(sl_top2_kernel<false>, at, (int)kTopSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sl_top2_kernel<true>, at, (int)kTopSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sl_resolve_tile_kernel, at, (int)kResSmemBytes);
    return e;
}

int launch_top2_pass(const SlArgs &a, cudaStream_t s) {
    if (!a.tgrid) return 0;
    launch_next(a.dump ? sl_top2_kernel<true> : sl_top2_kernel<false>, a.tgrid, kTopThreads, kTopSmemBytes, s, a);
    return 1;
}

int launch_top2_decide(const SlArgs &a, int sms, cudaStream_t s) {
    if (!a.npairs || !a.max_na) return 0;
    // four rows a thread once that still gives every SM its eight CTAs
    const bool four = a.n_rows >= 8ull * sms * 4 * kDecideThreads;
    const uint32_t rows = (four ? 4 : 1) * kDecideThreads, blocks = (uint32_t)(((uint64_t)a.max_na + rows - 1) / rows);
    int n = 0;
    for (uint32_t b = 0; b < blocks; b += 65535, ++n)  // a grid's second dimension: 67 M rows of one view
        launch_next(four ? sl_decide_kernel<4> : sl_decide_kernel<1>, dim3(a.npairs, std::min(65535u, blocks - b)),
                    kDecideThreads, 0, s, a, b);
    if (four) {
        launch_next(sl_nearest_kernel, 2 * sms, 256, 0, s, a);
        ++n;
    }
    return n;
}

int launch_top2_resolve(const SlArgs &a, int sms, cudaStream_t s) {
    if (!a.npairs || !a.max_na) return 0;
    SlArgs b = a;
    b.res_ctas = (uint32_t)std::min<uint64_t>(sms, a.n_tiles);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    // A group of 16 is a chain of dependent loads. With many groups (1 undecided row
    // in 100 assumed) they cover each other: four warps a group, four groups a
    // SM. With few, eight warps a CTA and the largest portable cluster that does
    // not exceed the GPU (one 8192 pair: 24 us against 93 with one CTA).
    const uint64_t est = a.n_rows / (100 * kGroupRows) + 1;
    const bool many = est >= (uint64_t)sms;
    uint32_t c = 1;
    while (!many && c < 8 && 2 * c * est <= 2ull * sms) c *= 2;
    at[0].val.clusterDim = {c, 1, 1};
    b.few_cluster = c;
    b.few_ctas = (uint32_t)((many ? 4 : 2) * sms) / c * c;
    cfg.gridDim = dim3(b.few_ctas);
    cfg.blockDim = dim3(many ? 128 : 256);
    cudaLaunchKernelEx(&cfg, sl_resolve_kernel, b);
    launch_next(sl_resolve_tile_kernel, b.res_ctas, kTopThreads, kResSmemBytes, s, b);
    return 2;
}

}  // namespace slm
