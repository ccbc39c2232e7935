// slm_internal.h — data layouts and kernel launchers shared by the host
// library (slm.cpp) and the CUDA translation units. Not part of the ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "slm.h"

namespace slm {

// Device error codes written to a launch's error word: a bounded wait gave up
// (TIMEOUT_*), or an invariant failed (BAD_ITEM: a work queue overflowed, a
// routing plan did not fit, a row was left undecided).
enum : uint32_t { DERR_NONE = 0, DERR_TIMEOUT_BAR = 1, DERR_BAD_ITEM = 2, DERR_TIMEOUT_MMA = 3 };

constexpr int kDesc = 128;      // descriptor length (features.rs:496)
constexpr int kTile = 128;      // rows per store tile
constexpr int kTileFloats = kTile * kDesc;

// Component k of a descriptor goes to slot perm(k) inside a store tile so that
// walking the slots in order walks the reference's accumulation order
// (matching.rs:146-155: lane k % 8, step k / 8): slot = (k % 8) * 16 + k / 8.
__host__ __device__ inline int perm_slot(int k) { return (k & 7) * 16 + (k >> 3); }

// Store tile layout (FP32): tile[slot][row], 128 x 128 floats = 64 KiB.

// Batches of at most this many pairs run their per-pair kernels (finalize,
// mid) with 1024 threads per pair instead of 256: with few pairs the GPU is
// not full and each pair's rows are a chain of dependent loads.
constexpr uint32_t kFewPairs = 64;

// Per-row partial state of an exact scan over a column range.
struct __align__(16) RowPart {
    float d1, d2;   // smallest and second smallest distance (multiset)
    uint32_t j1;    // lowest column index attaining d1 (0xffffffff: none)
    uint32_t pad;
};

#ifdef __CUDACC__
// Merges a column range's partial into a row state: (d1, lowest j1) and the
// second smallest of the multiset (matching.rs:182-187 applied per range).
__device__ __forceinline__ void merge_rowpart(const RowPart &p, float &d1, float &d2, uint32_t &j1) {
    const float nd2 = fminf(fmaxf(d1, p.d1), fminf(d2, p.d2));
    if (p.d1 < d1 || (p.d1 == d1 && p.j1 < j1)) {
        d1 = p.d1;
        j1 = p.j1;
    }
    d2 = nd2;
}
#endif

// Per image pair, as planned on the host.
struct PairMeta {
    uint32_t a_row0, b_row0;  // first store row of the two views (multiples of 128)
    uint32_t a_raw0, b_raw0;  // their first rows in the store's row-major array
    uint32_t na, nb;          // descriptor counts
    uint32_t nchunk;          // column chunks per row tile (exact path)
    uint32_t part_base;       // first RowPart block (128 rows per block)
    uint64_t col_base;        // first column-best entry
    uint64_t slot_off;        // first output slot (capacity na)
};

// One unit of the exact kernel: row groups [g0, g1) (of 32 rows, up to four) of
// the 128-row tile rt of pair `pair` against columns [32 q0, 32 q1) of b.
struct Item {
    uint32_t pair, rt, q0, q1;
    uint32_t part;  // RowPart block receiving the result (items of one tile and other rows share it)
    uint32_t g0, g1, pad;
};

struct ExactArgs {
    const float *tiled;          // FP32 store tiles
    const Item *items;
    uint32_t n_items;            // item capacity
    const uint32_t *n_items_dev; // if set, the item count is min(*n_items_dev, n_items), read on the device
    const PairMeta *pairs;
    RowPart *parts;
    unsigned long long *colbest; // (bits(d) << 32 | i), min-reduced
    uint32_t *work;              // dynamic item counter (zeroed per launch)
    uint32_t *err;               // device error word (zeroed per launch)
    int mutual;
    int x2;                      // 1: packed f32x2 arithmetic
    float zero;                  // 0.0f, read at run time: the addend of the packed squares
};

struct FinalizeArgs {
    const PairMeta *pairs;
    uint32_t npairs;
    const RowPart *parts;
    const unsigned long long *colbest;
    float ratio2;                // ratio * ratio in f32 (matching.rs:206)
    int mutual;
    uint2 *slots;                // output (i, j) slots
    uint32_t *counts;            // per-pair match count
    const uint32_t *err;         // if set: a count of 0xffffffff when this error word is set
};

// Pack n row-major descriptors (src, n x 128) into store tiles starting at
// tile index `tile0` (rows beyond n within the last tile are zeroed).
// The same for many views: tab holds one {row0, n, tile, view} per tile.
void launch_pack_fp32_tiles(const uint4 *tab, uint32_t ntiles, const float *raw, float *tiled, cudaStream_t s);
void launch_exact(const ExactArgs &a, int grid, cudaStream_t s);
// Sets kernel attributes (large shared memory) once per device; called at
// context creation, outside any stream capture. Fails if the kernel image
// cannot load on the device.
cudaError_t init_exact_kernels();
void launch_finalize(const FinalizeArgs &a, cudaStream_t s);
// One thread waits on a barrier that never completes for `polls` polls and
// records DERR_TIMEOUT_BAR in *err (self-test of the bounded waits).
void launch_wait_selftest(uint32_t polls, uint32_t *err, cudaStream_t s);
void launch_fill_u64(unsigned long long *p, uint64_t n, unsigned long long v, cudaStream_t s);
// Sets the message slm_last_error() returns on this host thread.
void set_last_error(const char *msg);

// Scratch layout of one exact FP32 pair match with its metadata made on the
// device (byte offsets; `inputs` adds room for copies of the row-major inputs).
constexpr uint32_t kSplitChunksMax = 16;  // finalize merges a row's chunks one after the other
inline uint32_t groups32(uint32_t n) { return (n + 31) / 32; }
// The shape of the items of a batch of few tiles (below two a SM): time counts
// rounds of the SMs, an item about 2.5 us and 1.55 us for each 32 x 32 block it
// holds, so a small batch gets small items and one of a tile a SM whole tiles.
// add() every pair, then the shape with the least time. One 317 x 300 pair's call
// took 54 us with whole tiles, 31 with single blocks; 1000 x 1000 rows 67 (before
// the kernels were launched early) and 48 (tiles' halves by rows), 1500 x 1500
// (144 tiles) 73 and 70.
struct ExactShape {
    uint32_t rows = 4, cols = 4;
};
struct ExactShapes {
    static constexpr ExactShape kShapes[6] = {{4, 4}, {2, 4}, {1, 4}, {2, 2}, {1, 2}, {1, 1}};
    uint64_t items[6] = {};
    uint32_t widest[6] = {};  // groups in the longest run of columns
    uint64_t tiles = 0;
    static uint32_t chunks_of(uint32_t nb, uint32_t cols) {
        const uint32_t n = (groups32(nb) + cols - 1) / cols;
        return n < 1 ? 1 : n > kSplitChunksMax ? kSplitChunksMax : n;
    }
    void add(uint32_t na, uint32_t nb) {
        tiles += (uint64_t)((na + kTile - 1) / kTile) * ((nb + kTile - 1) / kTile);
        for (int k = 0; k < 6; ++k) {
            const uint32_t chunks = chunks_of(nb, kShapes[k].cols), run = (groups32(nb) + chunks - 1) / chunks;
            items[k] += (uint64_t)((groups32(na) + kShapes[k].rows - 1) / kShapes[k].rows) * chunks;
            if (run > widest[k]) widest[k] = run;
        }
    }
    bool few(int sms) const { return tiles < 2ull * (uint64_t)sms; }
    ExactShape best(int sms) const {
        int at = 0;
        double least = 0;
        for (int k = 0; k < 6; ++k) {
            const double t = (double)((items[k] + sms - 1) / sms) * (2.5 + 1.55 * kShapes[k].rows * widest[k]);
            if (k == 0 || t < least) least = t, at = k;
        }
        return kShapes[at];
    }
};

struct SingleLayout {
    size_t tiled, items, parts, meta, colbest, slots, counts, ctl, raw_a, raw_b, bytes;
    uint32_t rt_n, ct_n, chunks;
    uint32_t rows, n_items;  // row groups of an item
    bool few;                // items of part of a tile (ExactShapes)
};
SingleLayout single_layout(uint32_t na, uint32_t nb, int sms, bool inputs);
// Whether finalize may write the match list straight into d_out: there must be
// room for every possible match (cap >= na), and finalize stores each pair as
// one 8-byte vector, while slm_pair itself only needs 4-byte alignment. Any
// other d_out gets the list through single_copy_kernel, which stores the two
// fields separately.
inline bool single_direct_output(const slm_pair *d_out, uint32_t cap, uint32_t na) {
    return cap >= na && (reinterpret_cast<uintptr_t>(d_out) & 7u) == 0;
}
// Enqueues the setup and packing, exact_kernel and finalize, which leave at
// most cap pairs in d_out and the count (0xffffffff: a device wait gave up) in
// *d_count (directly when single_direct_output holds, else through a copy
// kernel). Returns the launch status.
cudaError_t single_exact_enqueue(unsigned char *scratch, const SingleLayout &L, const float *d_a, uint32_t na,
                                 const float *d_b, uint32_t nb, float ratio, int mutual, slm_pair *d_out,
                                 uint32_t cap, uint32_t *d_count, int sms, cudaStream_t s);

// Sampson scoring of essential-matrix hypotheses (k_sampson.cu), all device
// pointers: pair p's matches are pts[pair_off[p] .. pair_off[p+1]) (a.x, a.y,
// b.x, b.y), hypothesis h is E[9 h .. 9 h + 9) (row-major) of pair
// hyp_pair[h]; counts[h] = #{i : |r| < thresh[p]}; with mask_off[h] !=
// ~0, the inlier bits at masks[mask_off[h] ..].
struct SampsonArgs {
    const double4 *pts;
    uint64_t n_pts;
    float4 *pts32;             // scratch of n_pts: the matches in f32
    const uint64_t *pair_off;
    const double *thresh;
    const double *E;
    const uint32_t *hyp_pair;
    uint64_t nh;
    uint32_t *counts;
    const uint64_t *mask_off;  // may be null (no masks)
    uint32_t *masks;
};
void launch_sampson(const SampsonArgs &a, cudaStream_t s);

// ---------------------------------------------------- descriptor producer
// (k_features.cu; crates/core/src/features.rs)

constexpr int kMaxBlurR = 127;  // blur radius ceil(3 sigma) the kernels take
constexpr int kMaxAngles = 18;  // local maxima of a 36-bin circular histogram

// Normalised taps of one gaussian_blur (features.rs:215-220), made on the host.
struct BlurTaps {
    float k[2 * kMaxBlurR + 1];
    int r;
};

// A refined DoG extremum that passed the contrast and edge tests.
struct __align__(16) FeatCand {
    float x, y;        // refined position in octave pixels
    float sig;         // sig_oct = sigma0 * kstep^s (s itself until launch_candidate_sigma)
    float value;       // refined DoG response
    uint16_t img;      // image of the batch
    uint8_t octave;
    uint8_t layer;     // refined layer (its gradient table)
    uint32_t pad;
    uint64_t key;      // emission order: octave << 48 | start layer << 32 | start y << 16 | start x
};

// One octave of a batch: its size and where its gradient tables start.
struct OctaveGeom {
    int w, h;
    uint64_t layer_stride;  // w * h
    uint64_t grad_off;      // float2 offset of (image 0, layer 1)
};

struct ExtremaArgs {
    const float *dog;       // [img][ng - 1][h][w]
    uint64_t layer_stride;
    int w, h, s, ng, octave;
    float contrast, edge_thr;
    FeatCand *cands;
    uint32_t *count;
    uint32_t cap;
};

struct OrientArgs {
    const FeatCand *cands;
    const uint32_t *count;
    uint32_t cap;
    const float2 *grads;    // every octave's tables: [img][layer 1..s][h][w] at geom.grad_off
    const OctaveGeom *geom;
    int s;
    float *angles;          // kMaxAngles per candidate
    uint8_t *nang;
    uint32_t few;           // launch_orient's: up to so many candidates have a CTA each
};

struct DescJob {
    uint32_t cand;          // candidate (or keypoint) index
    float angle;
    uint32_t out_row;       // descriptor row written
    uint32_t pad;
};

struct DescribeArgs {
    const DescJob *jobs;
    float2 *cs;             // scratch: cos and sin of each job's angle
    uint32_t n_large;       // the first jobs, those above describe_warp_side (all, with few features): a CTA each
    int max_side;           // the most window rows of any job (describe_side of the largest sigma)
    const FeatCand *cands;  // null: keypoints kps (image pixels) on one table, grads, geom[0]
    const slm_keypoint *kps;
    const float2 *grads;
    const OctaveGeom *geom;
    int s;
    float *desc;
};

cudaError_t init_feature_kernels();  // kernel attributes, once per device
// Both passes of a blur of nimg images (src -> tmp -> dst); with dog, also
// dog = dst - prev (prev strided as dst). Strides are per image, in floats.
void launch_blur(const float *src, float *tmp, float *dst, const float *prev, float *dog, int w, int h, int nimg,
                 uint64_t stride_src, uint64_t stride_dst, uint64_t stride_dog, const BlurTaps &t, int sms, cudaStream_t s);
void launch_downsample(const float *src, float *dst, int w, int h, int nimg, uint64_t stride_src,
                       uint64_t stride_dst, cudaStream_t s);
void launch_upsample2(const float *src, float *dst, int w, int h, int nimg, cudaStream_t s);
void launch_gray_from_rgb8(const uint8_t *rgb, float *out, uint64_t n, cudaStream_t s);
// n floats (whole groups of four) the device reads where they lie, 16-byte aligned
void launch_read_images(const float *src, float *dst, uint64_t n, int sms, cudaStream_t s);
// gradient tables of layers l0 .. l0 + s_ - 1 of each image (image k's layer l
// at gauss + k * img_stride + l * w * h); grad: [img][s_][h][w]
void launch_grad(const float *gauss, float2 *grad, int w, int h, int s_, uint64_t img_stride, int l0, int nimg,
                 cudaStream_t s);
// an octave's extrema, and the gradient tables of its layers 1 .. s (image k's layer
// l at gauss + k * img_stride + l * layer_stride)
void launch_layers(const ExtremaArgs &a, const float *gauss, float2 *grad, uint64_t img_stride, int nimg, int sms,
                   cudaStream_t s);
void launch_candidate_sigma(FeatCand *cands, const uint32_t *count, uint32_t cap, float sigma0, float kstep, int sms,
                            cudaStream_t s);
void launch_orient(const OrientArgs &a, int sms, cudaStream_t s);
constexpr int kDescWarpSide = 127;  // window rows one warp takes
// The window rows from which a feature gets a CTA instead of a warp: those a
// warp cannot take, or, with fewer features than four warps for each of the
// SMs' four sub-partitions, all: the chain of one warp then decides (one 717 x
// 531 photo's 1026 features 0.39 ms as warps, 0.13 as CTAs).
inline int describe_warp_side(size_t features, int sms) { return features < 16 * (size_t)sms ? 0 : kDescWarpSide; }
// Window rows of a feature of scale sigma (features.rs:526-528), at least.
inline int describe_side(float sigma) { return 2 * ((int)(3.0f * sigma * 1.41421356f * 2.5f + 0.5f) + 1) + 1; }
void launch_describe(const DescribeArgs &a, uint32_t njobs, cudaStream_t s);

// ------------------------------------------------------ tracks (k_tracks.cu)

struct TrackPair {  // slm_pair_matches
    uint32_t image_a, image_b;
    uint64_t first, count;
};

// Counters of one call (TrackArgs::ctl).
enum : int { kTrEdges, kTrInvalid, kTrMembers, kTrComps, kTrLarge, kTrConflicts, kTrShort, kTrTracks, kTrObs, kTrCount };
constexpr uint32_t kTrWarpMax = 256;  // members of a component one warp sorts

struct TrackArgs {
    const TrackPair *pairs;
    const uint2 *matches;     // (feature of image_a, feature of image_b)
    const uint32_t *nf;       // features per image
    const uint64_t *off;      // first node of each image, and the number of nodes
    uint32_t n_images;
    uint64_t n;               // nodes
    uint32_t min_length;
    unsigned long long *table;  // open-addressing edge set, all ones = empty
    uint64_t table_mask;      // slots - 1 (a power of two)
    unsigned long long *ctl;  // kTr* counters, zeroed
    // per node
    uint32_t *parent;
    uint8_t *used;            // has an edge
    uint32_t *cnt;            // of a root: members; after track_sort_kernel the track's length, or 0
    uint32_t *start;          // of a root: first of its members
    // per node with an edge, in component order
    uint32_t *members, *spare;  // spare may be parent's memory
    uint2 *sorted;            // members in order as (image, feature); may be the table's memory
    uint2 *comps;             // components {root, members}: small ones from the front, large from the back
    uint64_t max_comps;
    uint64_t share;           // nodes per CTA of the last two kernels, at most 1024 CTAs
    uint2 *sums;
    uint64_t *track_off;
    uint2 *obs;
};

// The whole of a call on the device: track_off, obs and the counters.
void launch_tracks(const TrackArgs &a, uint32_t n_pairs, int sms, cudaStream_t s);

}  // namespace slm
