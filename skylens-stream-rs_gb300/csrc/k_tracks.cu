// k_tracks.cu — the track builder's graph work on the GPU: build_tracks with
// ConflictPolicy::Drop (crates/core/src/tracks.rs:190-259) turns verified
// matches into edges between (image, feature) nodes and takes the connected
// components, each represented by its smallest node (tracks.rs:160-186:
// "the representative is always the smallest node", so the components and
// their representatives do not depend on the order the edges are joined in).
//
// Here: one CTA per image pair checks its matches (the reference's validity
// rule) and inserts each edge (small node << 32 | large node) into an
// open-addressing hash set, which counts the distinct edges. A new edge is
// hooked at once: the larger of its nodes' roots under the smaller, by one try in
// what the SM's cache holds of the parents. Wrong matches make one component of
// most nodes, and 1.7 M edges that each read its root from L2, or retry a
// compare-and-swap until it holds, took 0.6 to 2.8 ms; hooks that may fail,
// parents set to their roots, the edges hooked again, twice over, and a last pass
// that joins what is left take 0.07 ms after the edges' own kernel (0.21 ms: the
// matches are read from host memory, four a thread in flight). Then the
// components' members are gathered and sorted, the conflict and length rules
// applied, and the tracks laid out in root order, which is first-observation
// order: 0.05 ms, and the host sees finished lists. The call for the 1.7 M matches
// and 276 K nodes of a 240-view zone: 2.28 ms with a host synchronisation a round
// and the grouping on the host, now 0.34 ms, bound by latency of the matches' reads
// and of the hash set's atomics.
#include <cuda_runtime.h>

#include <cstdint>

#include "ptx.cuh"
#include "slm_internal.h"

namespace slm {

namespace {

constexpr unsigned long long kEmpty = ~0ull;

__device__ __forceinline__ uint64_t mix64(uint64_t x) {  // a 64-bit finaliser (xor-shift-multiply)
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}

// The root of x, in what the SM's cache holds of the parents: an ancestor of x in
// any case, but others may have hooked it since.
__device__ __forceinline__ uint32_t old_root(const uint32_t *parent, uint32_t x) {
    uint32_t p = parent[x];
    while (p != x) {
        x = p;
        p = parent[x];
    }
    return x;
}

__device__ __forceinline__ uint32_t find_root(const volatile uint32_t *parent, uint32_t x) {
    uint32_t p = parent[x];
    while (p != x) {
        x = p;
        p = parent[x];
    }
    return x;
}

// One try at joining the components of u and v. It may take a node for a root
// that is one no longer, and cut its link to an older parent: the edges are all
// looked at again until they are joined.
__device__ __forceinline__ void hook(uint32_t *parent, uint32_t u, uint32_t v) {
    const uint32_t ru = old_root(parent, u), rv = old_root(parent, v);
    if (ru != rv) atomicMin(parent + max(ru, rv), min(ru, rv));
}

// Joins the components of u and v: the larger root's parent becomes the
// smaller root. A root that lost its place meanwhile is looked up again (each
// such time another thread has joined two components).
__device__ __forceinline__ void join(uint32_t *parent, uint32_t u, uint32_t v) {
    if (old_root(parent, u) == old_root(parent, v)) return;
    for (;;) {
        u = find_root(parent, u);
        v = find_root(parent, v);
        if (u == v) return;
        const uint32_t big = max(u, v), small = min(u, v);
        if (atomicCAS(parent + big, big, small) == big) return;
    }
}

constexpr int kEdgeThreads = 256, kEdgeLoads = 4;

__global__ void __launch_bounds__(kEdgeThreads) track_edges_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    const TrackPair tp = a.pairs[blockIdx.x];
    const uint32_t ia = tp.image_a, ib = tp.image_b;
    const bool pair_ok = ia != ib && ia < a.n_images && ib < a.n_images;
    uint32_t bad = 0, fresh = 0;
    // four matches a thread in flight: they may lie in host memory (one at a time: 0.27 ms
    // of the zone's call against 0.12, without the hooks)
    for (uint64_t k0 = threadIdx.x; k0 < tp.count; k0 += kEdgeThreads * kEdgeLoads) {
        uint2 m[kEdgeLoads];
#pragma unroll
        for (int q = 0; q < kEdgeLoads; ++q)
            if (k0 + q * kEdgeThreads < tp.count) m[q] = a.matches[tp.first + k0 + q * kEdgeThreads];
#pragma unroll
        for (int q = 0; q < kEdgeLoads; ++q) {
            if (k0 + q * kEdgeThreads >= tp.count) break;
            if (!pair_ok || m[q].x >= a.nf[ia] || m[q].y >= a.nf[ib]) {
                ++bad;
                continue;
            }
            // the smaller image's node first (node = image offset + feature)
            const uint64_t u = a.off[ia] + m[q].x, v = a.off[ib] + m[q].y;
            const unsigned long long key = (u < v) ? (u << 32 | v) : (v << 32 | u);
            uint64_t slot = mix64(key) & a.table_mask;
            for (uint64_t probe = 0; probe <= a.table_mask; ++probe) {
                const unsigned long long prev = atomicCAS(&a.table[slot], kEmpty, key);
                if (prev == kEmpty) {  // a new edge
                    ++fresh;
                    a.used[u] = a.used[v] = 1;
                    hook(a.parent, (uint32_t)u, (uint32_t)v);
                    break;
                }
                if (prev == key) break;  // seen before
                slot = (slot + 1) & a.table_mask;
            }
        }
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    fresh = __reduce_add_sync(0xffffffffu, fresh);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicAdd(&a.ctl[kTrInvalid], (unsigned long long)bad);
        if (fresh) atomicAdd(&a.ctl[kTrEdges], (unsigned long long)fresh);
    }
}

// Every edge again; LAST: until it is joined.
template <bool LAST>
__global__ void __launch_bounds__(256) track_join_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    for (uint64_t x = blockIdx.x * 256ull + threadIdx.x; x <= a.table_mask; x += gridDim.x * 256ull) {
        const unsigned long long key = a.table[x];
        if (key == kEmpty) continue;
        const uint32_t u = (uint32_t)(key >> 32), v = (uint32_t)key;
        if constexpr (LAST)
            join(a.parent, u, v);
        else
            hook(a.parent, u, v);
    }
}

// Every node's parent becomes its root.
__global__ void __launch_bounds__(256) track_jump_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    for (uint64_t x = blockIdx.x * 256ull + threadIdx.x; x < a.n; x += gridDim.x * 256ull)
        a.parent[x] = old_root(a.parent, (uint32_t)x);
}

__global__ void __launch_bounds__(256) track_init_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    for (uint64_t x = blockIdx.x * 256ull + threadIdx.x; x < a.n; x += gridDim.x * 256ull) {
        a.parent[x] = (uint32_t)x;
        a.used[x] = 0;
        a.cnt[x] = 0;
    }
}

// Every node's root, and the members of each component (one atomic for the nodes
// of one root in a warp: wrong matches can make one component of most nodes). The walk writes nothing
// on its way: only x's own thread writes parent[x] here, so that it is the root
// when the kernel ends.
__global__ void __launch_bounds__(256) track_count_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    const volatile uint32_t *parent = a.parent;
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t x0 = blockIdx.x * 256ull + (threadIdx.x & ~31u); x0 < a.n; x0 += gridDim.x * 256ull) {  // warp-uniform
        const uint64_t x = x0 + lane;
        const bool used = x < a.n && a.used[x];
        uint32_t r = ~0u;  // no node
        if (used) {
            r = parent[x];
            for (uint32_t p = parent[r]; p != r; p = parent[r]) r = p;
            a.parent[x] = r;
        }
        const uint32_t same = __match_any_sync(0xffffffffu, r);
        if (used && lane == (uint32_t)__ffs(same) - 1) atomicAdd(&a.cnt[r], (uint32_t)__popc(same));
    }
}

// Room for each component's members, and the components' list: those that a
// warp sorts, and from the other end those that take a CTA.
__global__ void __launch_bounds__(256) track_list_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t x0 = blockIdx.x * 256ull + (threadIdx.x & ~31u); x0 < a.n; x0 += gridDim.x * 256ull) {  // warp-uniform
        const uint64_t x = x0 + lane;
        const uint32_t c = x < a.n ? a.cnt[x] : 0;
        uint32_t s = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        const uint32_t some = __ballot_sync(0xffffffffu, c != 0), big = __ballot_sync(0xffffffffu, c > kTrWarpMax);
        if (!some) continue;
        unsigned long long room = 0, listed = 0, large = 0;
        if (lane == 31) {
            room = atomicAdd(&a.ctl[kTrMembers], (unsigned long long)s);
            listed = atomicAdd(&a.ctl[kTrComps], (unsigned long long)__popc(some & ~big));
            if (big) large = atomicAdd(&a.ctl[kTrLarge], (unsigned long long)__popc(big));
        }
        room = __shfl_sync(0xffffffffu, room, 31);
        listed = __shfl_sync(0xffffffffu, listed, 31);
        large = __shfl_sync(0xffffffffu, large, 31);
        if (!c) continue;
        const uint32_t lt = (1u << lane) - 1, at = (uint32_t)(room + s - c);
        a.start[x] = at;
        const uint64_t k = c > kTrWarpMax ? a.max_comps - 1 - (large + __popc(big & lt)) : listed + __popc(some & ~big & lt);
        a.comps[k] = make_uint2((uint32_t)x, c);
    }
}

__global__ void __launch_bounds__(256) track_fill_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t x0 = blockIdx.x * 256ull + (threadIdx.x & ~31u); x0 < a.n; x0 += gridDim.x * 256ull) {  // warp-uniform
        const uint64_t x = x0 + lane;
        const bool used = x < a.n && a.used[x];
        const uint32_t r = used ? a.parent[x] : ~0u;
        const uint32_t same = __match_any_sync(0xffffffffu, r), first = __ffs(same) - 1;
        uint32_t left = 0;
        if (used && lane == first) left = atomicSub(&a.cnt[r], (uint32_t)__popc(same));
        left = __shfl_sync(0xffffffffu, left, first);
        if (used) a.members[a.start[r] + left - 1 - __popc(same & ((1u << lane) - 1))] = (uint32_t)x;
    }
}

// The image of node x: the last whose first node is at most x (images without
// features share their first node with the next).
__device__ __forceinline__ uint32_t image_of(const TrackArgs &a, uint32_t x) {
    uint32_t lo = 0, hi = a.n_images;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (a.off[mid] <= x)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// The observation of node x; conflict: another member y of its component lies
// in the same image.
struct Seat {
    uint32_t img;
    uint64_t lo, hi;  // the image's nodes
};
__device__ __forceinline__ Seat seat_of(const TrackArgs &a, uint32_t x) {
    const uint32_t img = image_of(a, x);
    return Seat{img, a.off[img], a.off[img + 1]};
}

__device__ __forceinline__ void finish_component(const TrackArgs &a, uint32_t root, uint32_t len, bool bad) {
    if (bad)
        atomicAdd(&a.ctl[kTrConflicts], 1ull);
    else if (len < a.min_length)
        atomicAdd(&a.ctl[kTrShort], 1ull);
    else
        a.cnt[root] = len;
}

// A component of up to kTrWarpMax nodes by one warp: a member's place is the
// number of smaller ones.
__device__ __forceinline__ void sort_small(const TrackArgs &a, uint32_t root, uint32_t len, uint32_t lane) {
    const uint32_t *in = a.members + a.start[root];
    uint2 *out = a.sorted + a.start[root];
    bool bad = len > a.n_images;  // more members than images
    for (uint32_t k = lane; k < len; k += 32) {
        const uint32_t x = in[k];
        const Seat s = seat_of(a, x);
        uint32_t place = 0;
        for (uint32_t q = 0; q < len; ++q) {
            const uint32_t y = in[q];
            place += y < x;
            bad |= y != x && y >= s.lo && y < s.hi;
        }
        out[place] = make_uint2(s.img, (uint32_t)(x - s.lo));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) finish_component(a, root, len, bad);
}

// A larger one by a CTA: merges of runs of 1, 2, 4... members between two
// buffers, each member's place in the merged run by binary search in the other.
__device__ __forceinline__ void sort_large(const TrackArgs &a, uint32_t root, uint32_t len) {
    bool bad = len > a.n_images;
    if (!bad) {
        uint32_t *in = a.members + a.start[root], *out = a.spare + a.start[root];
        for (uint64_t w = 1; w < len; w *= 2) {
            for (uint64_t k = threadIdx.x; k < len; k += 256) {
                const uint32_t x = in[k];
                const uint64_t r = k / w, other = (r ^ 1) * w;
                uint64_t lo = other, hi = min(other + w, (uint64_t)len);
                while (lo < hi) {
                    const uint64_t mid = (lo + hi) / 2;
                    if (in[mid] < x)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                out[other < len ? (r & ~1ull) * w + (k - r * w) + (lo - other) : k] = x;
            }
            __syncthreads();
            uint32_t *t = in;
            in = out, out = t;
        }
        for (uint64_t k = threadIdx.x; k < len; k += 256) {
            const uint32_t x = in[k];
            const Seat s = seat_of(a, x);
            bad |= k && in[k - 1] >= s.lo;  // smaller, and in the same image
            a.sorted[a.start[root] + k] = make_uint2(s.img, (uint32_t)(x - s.lo));
        }
    }
    bad = __syncthreads_or(bad) != 0;
    if (threadIdx.x == 0) finish_component(a, root, len, bad);
}

__global__ void __launch_bounds__(256) track_sort_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n = a.ctl[kTrComps], large = a.ctl[kTrLarge];
    for (uint64_t k = blockIdx.x * 8ull + (threadIdx.x >> 5); k < n; k += gridDim.x * 8ull) {  // warp-uniform
        const uint2 c = a.comps[k];
        sort_small(a, c.x, c.y, lane);
    }
    for (uint64_t k = blockIdx.x; k < large; k += gridDim.x) {  // block-uniform
        const uint2 c = a.comps[a.max_comps - 1 - k];
        sort_large(a, c.x, c.y);
    }
}

// Tracks and observations of each CTA's share of the nodes.
__global__ void __launch_bounds__(256) track_sums_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    __shared__ uint32_t ws[2][8];
    const uint64_t x0 = blockIdx.x * a.share, x1 = min(x0 + a.share, a.n);
    uint32_t t = 0, o = 0;
    for (uint64_t x = x0 + threadIdx.x; x < x1; x += 256) {
        const uint32_t c = a.cnt[x];
        t += c != 0;
        o += c;
    }
    t = __reduce_add_sync(0xffffffffu, t);
    o = __reduce_add_sync(0xffffffffu, o);
    if ((threadIdx.x & 31) == 0) ws[0][threadIdx.x >> 5] = t, ws[1][threadIdx.x >> 5] = o;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) t += ws[0][w], o += ws[1][w];
        a.sums[blockIdx.x] = make_uint2(t, o);
    }
}

// Their lists, in root order: track k is obs[track_off[k] .. track_off[k + 1]).
__global__ void __launch_bounds__(256) track_emit_kernel(TrackArgs a) {
    grid_wait();
    grid_go();
    __shared__ uint32_t ws[2][8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto total = [&](uint32_t t, uint32_t o, uint32_t &pt, uint32_t &po, uint32_t &at, uint32_t &ao) {  // scan of (t, o)
        pt = t, po = o;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, pt, k), v = __shfl_up_sync(0xffffffffu, po, k);
            if (lane >= k) pt += u, po += v;
        }
        __syncthreads();
        if (lane == 31) ws[0][warp] = pt, ws[1][warp] = po;
        __syncthreads();
        at = ao = 0;
        for (uint32_t w = 0; w < 8; ++w) {
            if (w < warp) pt += ws[0][w], po += ws[1][w];
            at += ws[0][w], ao += ws[1][w];
        }
        pt -= t, po -= o;  // exclusive
    };
    uint32_t t = 0, o = 0, pt, po, at, ao;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += 256) t += a.sums[b].x, o += a.sums[b].y;
    uint32_t t0, o0;
    total(t, o, pt, po, t0, o0);  // tracks and observations before this CTA's share
    const uint64_t x0 = blockIdx.x * a.share, x1 = min(x0 + a.share, a.n);
    for (uint64_t base = x0; base < x1; base += 256) {
        const uint64_t x = base + threadIdx.x;
        const uint32_t c = x < x1 ? a.cnt[x] : 0;
        total(c != 0, c, pt, po, at, ao);
        if (c) a.track_off[t0 + pt] = o0 + po;
        const uint32_t from = c ? a.start[x] : 0;
        for (uint32_t todo = __ballot_sync(0xffffffffu, c != 0); todo; todo &= todo - 1) {  // a warp per track
            const int l = __ffs(todo) - 1;
            const uint32_t len = __shfl_sync(0xffffffffu, c, l), src = __shfl_sync(0xffffffffu, from, l),
                           dst = o0 + __shfl_sync(0xffffffffu, po, l);
            for (uint32_t q = lane; q < len; q += 32) a.obs[dst + q] = a.sorted[src + q];
        }
        t0 += at, o0 += ao;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        a.track_off[t0] = o0;
        a.ctl[kTrTracks] = t0;
        a.ctl[kTrObs] = o0;
    }
}

}  // namespace

void launch_tracks(const TrackArgs &a, uint32_t n_pairs, int sms, cudaStream_t s) {
    const int grid = 8 * sms;
    launch_next(track_init_kernel, grid, 256, 0, s, a);
    if (n_pairs) launch_next(track_edges_kernel, n_pairs, kEdgeThreads, 0, s, a);
    for (int round = 0; round < 2; ++round) {
        launch_next(track_jump_kernel, grid, 256, 0, s, a);
        launch_next(track_join_kernel<false>, grid, 256, 0, s, a);
    }
    launch_next(track_jump_kernel, grid, 256, 0, s, a);
    launch_next(track_join_kernel<true>, grid, 256, 0, s, a);
    launch_next(track_count_kernel, grid, 256, 0, s, a);
    launch_next(track_list_kernel, grid, 256, 0, s, a);
    launch_next(track_fill_kernel, grid, 256, 0, s, a);
    launch_next(track_sort_kernel, grid, 256, 0, s, a);
    const unsigned blocks = a.n ? (unsigned)((a.n + a.share - 1) / a.share) : 1u;
    launch_next(track_sums_kernel, blocks, 256, 0, s, a);
    launch_next(track_emit_kernel, blocks, 256, 0, s, a);
}

}  // namespace slm
