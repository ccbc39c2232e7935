// k_features.cu — the descriptor producer on the GPU: Gaussian pyramid, DoG
// extrema with sub-pixel refinement, orientation assignment and the 128-d
// descriptor of crates/core/src/features.rs (detect_core :650-781,
// gaussian_blur :214-250, pixel_grad :327-332, orientations_with :361-420,
// refine_extremum :431-484, describe_with :521-592), over a batch of images
// of one size.
//
// Every arithmetic expression keeps the reference's operand order; the file
// is compiled without FMA contraction and with IEEE division and square root,
// so each f32 value is the reference's. The reference's per-pixel and
// per-keypoint transcendental functions (atan2, exp, powf, cos, sin; the
// platform's float functions) are evaluated correctly rounded: atan2 and exp,
// called per pixel and per window sample, by the float-float evaluations of
// fmath_cr.h (FP32 and FMA, with a rounding test that falls back to double in
// a few calls in 10^5), powf, cos and sin, once per keypoint, in double
// rounded to float. Both equal the double function rounded to float (double
// rounding aside, probability about 2^-29 a call), which equals the
// platform's float result wherever that one is correctly rounded. Sums that
// the reference accumulates in one order (histogram bins, the descriptor's
// norm) are accumulated in that order.
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "fmath_cr.h"
#include "ptx.cuh"
#include "slm_internal.h"

namespace slm {

namespace {

constexpr float kTwoPi = 6.28318530717958647692f;  // std::f32::consts::TAU
constexpr float kSqrt2 = 1.41421356237309504880f;  // std::f32::consts::SQRT_2
constexpr int kOriBins = 36;                        // features.rs:307

__device__ __forceinline__ float exp_cr(float x) { return slm_expf_neg_cr(x); }
__device__ __forceinline__ float atan2_cr(float y, float x) { return slm_atan2f_cr(y, x); }

// f32::rem_euclid(a, b) for b > 0: a % b (fmodf), plus b when negative. For
// |a| < 2b the remainder is a, or a - b with a's sign (exact: b <= |a| < 2b),
// and a zero remainder keeps a's sign as fmodf's does; fmodf otherwise.
__device__ __forceinline__ float rem_euclid(float a, float b) {
    float r;
    const float aa = fabsf(a);
    if (aa < b) {
        r = a;
    } else if (aa < 2.0f * b) {
        r = copysignf(aa - b, a);
    } else {
        r = fmodf(a, b);
    }
    return r < 0.0f ? r + b : r;
}

// `v as isize` (truncation; the values here are small and finite)
__device__ __forceinline__ int f2i(float v) { return v != v ? 0 : (int)v; }

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : v > hi ? hi : v; }

// ------------------------------------------------------------------ blur

constexpr int kBlurX = 256;

// Horizontal pass: tmp[y][x] = sum_j k[j] * src[y][clamp(x + j - r)], j in
// order, starting from 0.0 (features.rs:226-238).
__global__ void __launch_bounds__(kBlurX) blur_rows_kernel(const float *__restrict__ src, float *__restrict__ dst,
                                                           int w, int h, uint64_t img_stride_src,
                                                           uint64_t img_stride_dst, BlurTaps t) {
    __shared__ float row[kBlurX + 2 * kMaxBlurR];
    const int y = grid_wait(blockIdx.y), b = blockIdx.z;
    const int x0 = blockIdx.x * kBlurX;
    const float *s = src + b * img_stride_src + (uint64_t)y * w;
    const int n = kBlurX + 2 * t.r;
    for (int i = threadIdx.x; i < n; i += kBlurX) row[i] = s[clampi(x0 + i - t.r, 0, w - 1)];
    __syncthreads();
    const int x = x0 + threadIdx.x;
    if (x >= w) return;
    float acc = 0.0f;
    for (int j = 0; j <= 2 * t.r; ++j) acc += t.k[j] * row[threadIdx.x + j];
    dst[b * img_stride_dst + (uint64_t)y * w + x] = acc;
}

// Vertical pass: out[y][x] = sum_j k[j] * tmp[clamp(y + j - r)][x], j in
// order from 0.0 (features.rs:240-249); with `prev`, also the DoG layer
// out - prev (features.rs:674-685).
__global__ void __launch_bounds__(kBlurX) blur_cols_kernel(const float *__restrict__ tmp, float *__restrict__ out,
                                                           const float *__restrict__ prev, float *__restrict__ dog,
                                                           int w, int h, uint64_t img_stride_tmp,
                                                           uint64_t img_stride_out, uint64_t img_stride_dog,
                                                           BlurTaps t) {
    const int x = blockIdx.x * kBlurX + threadIdx.x, y = grid_wait(blockIdx.y), b = blockIdx.z;
    if (x >= w) return;
    const float *c = tmp + b * img_stride_tmp + x;
    float acc = 0.0f;
    for (int j = 0; j <= 2 * t.r; ++j) acc += t.k[j] * c[(uint64_t)clampi(y + j - t.r, 0, h - 1) * w];
    const uint64_t p = (uint64_t)y * w + x;
    out[b * img_stride_out + p] = acc;
    if (dog) dog[b * img_stride_dog + p] = acc - prev[b * img_stride_out + p];
}

// Both passes in one kernel for radii up to kFusedR: a 64 x 32 output tile
// with its halo of clamped input pixels in shared memory, the horizontal sums
// of the tile's rows (halo rows included) in shared memory, then the vertical
// sums; with `dog`, also dog = out - src at each pixel (src is the previous
// layer). Each sum runs over j in order from 0.0, exactly as the two-kernel
// form and the reference do.
// Bound by instruction issue, so a thread computes 8 neighbouring sums from the
// 8 + 2 R values they share, in registers (the radius is a template argument):
// one shared load for three to five multiply-adds instead of one for each.
// 1.10 -> 0.58 ms for the six layers of 24 views of 960 x 540 and their octaves.
// Row pitches are 4 modulo 32 words: 8 lanes reading 16 bytes each of
// consecutive rows cover all banks once.
constexpr int kFusedR = 16;
constexpr int kFX = 64, kFRun = 8;
constexpr int kFInPitch = 100, kFSumPitch = 68;
static_assert(kFX + 2 * kFusedR <= kFInPitch && kFInPitch % 32 == 4 && kFSumPitch % 32 == 4, "tile pitches");

// Output rows of a tile: with its halo 64 rows or a few less (TALL), so that
// the horizontal sums keep every thread busy twice, or 32.
template <int R, bool TALL>
__host__ __device__ constexpr int blur_rows() {
    return TALL ? (64 - 2 * R) / 4 * 4 : 32;
}
template <int R, bool TALL>
__host__ __device__ constexpr size_t blur_smem() {
    return sizeof(float) * (size_t)(blur_rows<R, TALL>() + 2 * R) * (kFInPitch + kFSumPitch);
}

template <int R, bool TALL>
__global__ void __launch_bounds__(256) blur_fused_kernel(const float *__restrict__ src, float *__restrict__ dst,
                                                         float *__restrict__ dog, int w, int h,
                                                         uint64_t img_stride_src, uint64_t img_stride_dst,
                                                         uint64_t img_stride_dog, BlurTaps t) {
    extern __shared__ __align__(16) float blur_tile[];
    constexpr int kFY = blur_rows<R, TALL>(), rows = kFY + 2 * R, cols = kFX + 2 * R, N = kFRun + 2 * R;
    constexpr int V = kFY / 4;  // a column's run: 64 columns x 4 runs = 256 threads
    float *in = blur_tile, *hs = blur_tile + rows * kFInPitch;
    const int b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x0 = blockIdx.x * kFX, y0 = grid_wait(blockIdx.y) * kFY;
    grid_go();
    const float *S = src + b * img_stride_src;
#pragma unroll 4
    for (int ry = warp; ry < rows; ry += 8) {
        const float *line = S + (uint64_t)clampi(y0 + ry - R, 0, h - 1) * w;
#pragma unroll
        for (int c = 0; c < cols; c += 32)
            if (c + lane < cols) in[ry * kFInPitch + c + lane] = line[clampi(x0 + c + lane - R, 0, w - 1)];
    }
    __syncthreads();
    // a run of 8 sums of one row a thread, consecutive lanes on consecutive rows
    for (int e = threadIdx.x; e < rows * (kFX / kFRun); e += 256) {
        const int ry = e % rows, cx = e / rows * kFRun;
        float v[(N + 3) / 4 * 4];
#pragma unroll
        for (int k = 0; k < (N + 3) / 4; ++k) {
            const float4 f = *reinterpret_cast<const float4 *>(&in[ry * kFInPitch + cx + 4 * k]);
            v[4 * k] = f.x, v[4 * k + 1] = f.y, v[4 * k + 2] = f.z, v[4 * k + 3] = f.w;
        }
        float acc[kFRun];
#pragma unroll
        for (int k = 0; k < kFRun; ++k) {
            acc[k] = 0.0f;
#pragma unroll
            for (int j = 0; j <= 2 * R; ++j) acc[k] += t.k[j] * v[k + j];
        }
        float4 *o = reinterpret_cast<float4 *>(&hs[ry * kFSumPitch + cx]);
        o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    }
    __syncthreads();
    // a run of V sums of one column a thread
    const int cx = threadIdx.x % kFX, ty = threadIdx.x / kFX * V, x = x0 + cx;
    if (x >= w) return;
    float v[V + 2 * R];
#pragma unroll
    for (int k = 0; k < V + 2 * R; ++k) v[k] = hs[(ty + k) * kFSumPitch + cx];
#pragma unroll
    for (int k = 0; k < V; ++k) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j <= 2 * R; ++j) acc += t.k[j] * v[k + j];
        const int y = y0 + ty + k;
        if (y < h) {
            const uint64_t p = (uint64_t)y * w + x;
            dst[b * img_stride_dst + p] = acc;
            if (dog) dog[b * img_stride_dog + p] = acc - in[(ty + k + R) * kFInPitch + cx + R];
        }
    }
}

// base of the next octave: the even pixels of gauss[s] (GrayImage::downsample)
__global__ void downsample_kernel(const float *__restrict__ src, float *__restrict__ dst, int w, int h, int nw, int nh,
                                  uint64_t img_stride_src, uint64_t img_stride_dst) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = grid_wait(blockIdx.y), b = blockIdx.z;
    grid_go();
    if (x >= nw) return;
    dst[b * img_stride_dst + (uint64_t)y * nw + x] = src[b * img_stride_src + (uint64_t)(2 * y) * w + 2 * x];
}

// GrayImage::upsample2 (features.rs:62-85): bilinear at pixel centres.
__global__ void upsample2_kernel(const float *__restrict__ src, float *__restrict__ dst, int w, int h) {
    const int W = 2 * w;
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = grid_wait(blockIdx.y), b = blockIdx.z;
    grid_go();
    if (x >= W) return;
    const float *s = src + (uint64_t)b * w * h;
    const float sy = ((float)y + 0.5f) / 2.0f - 0.5f;
    const float y0 = floorf(sy), fy = sy - y0;
    const int ya = clampi(f2i(y0), 0, h - 1), yb = clampi(f2i(y0) + 1, 0, h - 1);
    const float sx = ((float)x + 0.5f) / 2.0f - 0.5f;
    const float x0 = floorf(sx), fx = sx - x0;
    const int xa = clampi(f2i(x0), 0, w - 1), xb = clampi(f2i(x0) + 1, 0, w - 1);
    const float top = s[(uint64_t)ya * w + xa] * (1.0f - fx) + s[(uint64_t)ya * w + xb] * fx;
    const float bot = s[(uint64_t)yb * w + xa] * (1.0f - fx) + s[(uint64_t)yb * w + xb] * fx;
    dst[(uint64_t)b * W * (2 * h) + (uint64_t)y * W + x] = top * (1.0f - fy) + bot * fy;
}

// GrayImage::from_rgb (features.rs:165-189). Four pixels a thread where the
// bytes lie on a 4-byte boundary: three word loads, one 16-byte store.
__device__ __forceinline__ float gray_of(uint32_t r, uint32_t g, uint32_t b) {
    return (0.299f * (float)r + 0.587f * (float)g + 0.114f * (float)b) / 255.0f;
}
__global__ void __launch_bounds__(256) gray_from_rgb8_kernel(const uint8_t *rgb, float *out, uint64_t n, bool wide) {
    grid_wait();
    grid_go();
    const uint64_t i = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * 4;
    if (wide && i + 4 <= n) {
        const uint32_t *c = reinterpret_cast<const uint32_t *>(rgb + 3 * i);
        const uint32_t u = c[0], v = c[1], t = c[2];
        *reinterpret_cast<float4 *>(out + i) =
            make_float4(gray_of(u & 255, u >> 8 & 255, u >> 16 & 255), gray_of(u >> 24, v & 255, v >> 8 & 255),
                        gray_of(v >> 16 & 255, v >> 24, t & 255), gray_of(t >> 8 & 255, t >> 16 & 255, t >> 24));
        return;
    }
    for (uint64_t k = i; k < n && k < i + 4; ++k) out[k] = gray_of(rgb[3 * k], rgb[3 * k + 1], rgb[3 * k + 2]);
}

// Images that lie in host memory the device reads where it is: one read over
// the link, 16 bytes a thread.
__global__ void __launch_bounds__(256) read_images_kernel(const float4 *src, float4 *dst, uint64_t n4) {
    grid_wait();
    grid_go();
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += (uint64_t)gridDim.x * 256) dst[i] = src[i];
}

// GradTable (features.rs:335-359) of s consecutive layers from l0: |g| and
// atan2(gy, gx) of central differences at interior pixels (pixel_grad,
// :327-332); grad is [img][s][h][w]. Bound by instruction issue (the atan2 and
// the square root): a thread walks kGradRows rows of a column, so that address
// arithmetic and two of a pixel's four loads are shared. 0.49 -> 0.30 ms for the
// octaves of 24 views of 960 x 540, the atan2's part of it included.
constexpr int kGradRows = 6;
constexpr int kGradThreads = 128;
__device__ __forceinline__ void grad_tile(const float *__restrict__ gauss, float2 *__restrict__ grad, int w, int h, int s,
                                          uint64_t layer_stride, uint64_t img_stride, int l0, uint3 block) {
    const int x = block.x * kGradThreads + threadIdx.x, y0 = block.y * kGradRows;
    const int b = block.z / s, l = block.z % s;
    if (x >= w) return;
    const bool inside = x >= 1 && x + 1 < w;
    const float *im = gauss + (uint64_t)b * img_stride + (uint64_t)(l0 + l) * layer_stride + (uint64_t)y0 * w + x;
    float2 *out = grad + ((uint64_t)b * s + l) * layer_stride + (uint64_t)y0 * w + x;
    float above = inside && y0 >= 1 ? im[-w] : 0.0f, here = im[0];
#pragma unroll
    for (int k = 0; k < kGradRows; ++k, im += w, out += w) {
        const int y = y0 + k;
        if (y >= h) return;
        const float below = y + 1 < h ? im[w] : 0.0f;
        float2 g = make_float2(0.0f, 0.0f);
        if (inside && y >= 1 && y + 1 < h) {
            const float gx = im[1] - im[-1];
            const float gy = below - above;
            g.x = sqrtf(gx * gx + gy * gy);
            g.y = atan2_cr(gy, gx);
        }
        *out = g;
        above = here;
        here = below;
    }
}

__global__ void __launch_bounds__(kGradThreads) grad_kernel(const float *__restrict__ gauss, float2 *__restrict__ grad,
                                                            int w, int h, int s, uint64_t layer_stride,
                                                            uint64_t img_stride, int l0) {
    const uint32_t y = grid_wait(blockIdx.y);
    grid_go();
    grad_tile(gauss, grad, w, h, s, layer_stride, img_stride, l0, make_uint3(blockIdx.x, y, blockIdx.z));
}

// ---------------------------------------------------------------- extrema

// nalgebra 0.33 Matrix3::try_inverse (cofactor formula), m row-major;
// false when the determinant is exactly zero.
__device__ bool inverse3(const float (&m)[9], float (&o)[9]) {
    const float m11 = m[0], m12 = m[1], m13 = m[2];
    const float m21 = m[3], m22 = m[4], m23 = m[5];
    const float m31 = m[6], m32 = m[7], m33 = m[8];
    const float minor_m12_m23 = m22 * m33 - m32 * m23;
    const float minor_m11_m23 = m21 * m33 - m31 * m23;
    const float minor_m11_m22 = m21 * m32 - m31 * m22;
    const float det = m11 * minor_m12_m23 - m12 * minor_m11_m23 + m13 * minor_m11_m22;
    if (det == 0.0f) return false;
    o[0] = minor_m12_m23 / det;
    o[1] = (m13 * m32 - m33 * m12) / det;
    o[2] = (m12 * m23 - m22 * m13) / det;
    o[3] = -minor_m11_m23 / det;
    o[4] = (m11 * m33 - m31 * m13) / det;
    o[5] = (m13 * m21 - m23 * m11) / det;
    o[6] = minor_m11_m22 / det;
    o[7] = (m12 * m31 - m32 * m11) / det;
    o[8] = (m11 * m22 - m21 * m12) / det;
    return true;
}

// max and min of three that are NaN when an operand is: v > max_nan(...) is
// then false, as the reference's comparison with that operand is.
__device__ __forceinline__ float max3n(float a, float b, float c) {
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3n(float a, float b, float c) {
    float d;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ void refine_candidate(const ExtremaArgs &a, const float *dog, int b, int l0, int x, int y);

// detect_core's scan (features.rs:700-768) over the interior pixels of DoG
// layers 1..s: contrast, the 26-neighbour test, then refine_candidate for the
// few that pass. Bound by the 27 loads a pixel would take: a lane has a column
// (30 of a warp's 32 lanes test theirs, the outer two serve their neighbours),
// walks down a strip of rows and loads each row's pixel of the three layers
// once; the maxima and minima of its column's nine values go to both sides by
// shuffle. The extrema, a few in a thousand pixels, wait in shared memory until
// the CTA's strips are through and are then refined side by side instead of one
// lane at a time. 0.49 -> 0.23 ms for the octaves of 24 views of 960 x 540.
constexpr int kExtremaWarps = 4, kExtremaRows = 16;
__device__ __forceinline__ void extrema_strips(const ExtremaArgs &a, int rows, uint3 block) {
    // no two maxima, and no two minima, are neighbours: at most one of each in 2 x 2 pixels
    __shared__ uint32_t found[30 * kExtremaRows * kExtremaWarps / 2];
    __shared__ uint32_t n_found;
    if (threadIdx.x == 0) n_found = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, strip = block.y * kExtremaWarps + (threadIdx.x >> 5);
    const int b = block.z / a.s, l0 = 1 + block.z % a.s;
    const int w = a.w, h = a.h;
    const int x = (int)block.x * 30 + lane, y0 = 1 + strip * rows;  // lanes 1 .. 30 test pixel x
    const float *dog = a.dog + (uint64_t)b * (a.ng - 1) * a.layer_stride;
    if (y0 < h - 1) {  // warp-uniform
        const float *lo = dog + (uint64_t)(l0 - 1) * a.layer_stride + min(x, w - 1);
        const float *mid = lo + a.layer_stride, *up = mid + a.layer_stride;
        const bool mine = lane >= 1 && lane <= 30 && x + 1 < w;
        uint64_t row = (uint64_t)(y0 - 1) * w;
        float l1 = lo[row], m1 = mid[row], u1 = up[row];  // rows y - 1, y, y + 1 of the three layers
        row += w;
        float l2 = lo[row], m2 = mid[row], u2 = up[row];
        const int end = min(y0 + rows, h - 1);
        for (int y = y0; y < end; ++y) {
            row += w;
            const float l3 = lo[row], m3 = mid[row], u3 = up[row];
            // the column's values but the pixel itself, then with it for the neighbours
            const float mxo = max3n(max3n(l1, l2, l3), max3n(u1, u2, u3), max3n(m1, m3, m3));
            const float mno = min3n(min3n(l1, l2, l3), min3n(u1, u2, u3), min3n(m1, m3, m3));
            const float mx = max3n(mxo, m2, m2), mn = min3n(mno, m2, m2);
            const float mxs = max3n(__shfl_up_sync(0xffffffffu, mx, 1), __shfl_down_sync(0xffffffffu, mx, 1), mxo);
            const float mns = min3n(__shfl_up_sync(0xffffffffu, mn, 1), __shfl_down_sync(0xffffffffu, mn, 1), mno);
            if (mine && !(fabsf(m2) < a.contrast) && (m2 > mxs || m2 < mns))
                found[atomicAdd(&n_found, 1u)] = (uint32_t)y << 16 | (uint32_t)x;
            l1 = l2, l2 = l3, m1 = m2, m2 = m3, u1 = u2, u2 = u3;
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < n_found; k += 32 * kExtremaWarps)
        refine_candidate(a, dog, b, l0, (int)(found[k] & 0xffffu), (int)(found[k] >> 16));
}

// refine_extremum, the contrast and edge tests; a survivor is appended to the
// candidate list with its emission-order key.
__device__ void refine_candidate(const ExtremaArgs &a, const float *dog, int b, int l0, int x, int y) {
    const int w = a.w, h = a.h;
#define D(L, X, Y) dog[(uint64_t)(L) * a.layer_stride + (uint64_t)(Y) * w + (X)]
    // refine_extremum (features.rs:431-484)
    int cx = x, cy = y, cl = l0;
    bool ok = false;
    float d[3], g[3], v = 0.0f;
    for (int it = 0; it < 5; ++it) {
        v = D(cl, cx, cy);
        g[0] = 0.5f * (D(cl, cx + 1, cy) - D(cl, cx - 1, cy));
        g[1] = 0.5f * (D(cl, cx, cy + 1) - D(cl, cx, cy - 1));
        g[2] = 0.5f * (D(cl + 1, cx, cy) - D(cl - 1, cx, cy));
        const float hxx = D(cl, cx + 1, cy) + D(cl, cx - 1, cy) - 2.0f * v;
        const float hyy = D(cl, cx, cy + 1) + D(cl, cx, cy - 1) - 2.0f * v;
        const float hss = D(cl + 1, cx, cy) + D(cl - 1, cx, cy) - 2.0f * v;
        const float hxy = 0.25f * (D(cl, cx + 1, cy + 1) - D(cl, cx - 1, cy + 1) - D(cl, cx + 1, cy - 1) +
                                   D(cl, cx - 1, cy - 1));
        const float hxs = 0.25f * (D(cl + 1, cx + 1, cy) - D(cl + 1, cx - 1, cy) - D(cl - 1, cx + 1, cy) +
                                   D(cl - 1, cx - 1, cy));
        const float hys = 0.25f * (D(cl + 1, cx, cy + 1) - D(cl + 1, cx, cy - 1) - D(cl - 1, cx, cy + 1) +
                                   D(cl - 1, cx, cy - 1));
        const float hm[9] = {hxx, hxy, hxs, hxy, hyy, hys, hxs, hys, hss};
        float inv[9];
        if (!inverse3(hm, inv)) return;
#pragma unroll
        for (int i = 0; i < 3; ++i) {  // matrix x vector: columns added in order (gemv)
            float acc = inv[3 * i] * g[0];
            acc = acc + inv[3 * i + 1] * g[1];
            acc = acc + inv[3 * i + 2] * g[2];
            d[i] = -acc;
        }
        if (fabsf(d[0]) <= 0.5f && fabsf(d[1]) <= 0.5f && fabsf(d[2]) <= 0.5f) {
            ok = true;
            break;
        }
        if (!(isfinite(d[0]) && isfinite(d[1]) && isfinite(d[2]))) return;
        const int nx = cx + f2i(roundf(d[0])), ny = cy + f2i(roundf(d[1])), nl = cl + f2i(roundf(d[2]));
        if (nx < 1 || ny < 1 || nl < 1 || nx >= w - 1 || ny >= h - 1 || nl > a.s) return;
        cx = nx;
        cy = ny;
        cl = nl;
    }
    if (!ok) return;
    const float value = v + 0.5f * (g[0] * d[0] + g[1] * d[1] + g[2] * d[2]);
    if (fabsf(value) < a.contrast) return;
    // edge test on the refined sample (features.rs:735-746)
    const float c = D(cl, cx, cy);
    const float dxx = D(cl, cx + 1, cy) + D(cl, cx - 1, cy) - 2.0f * c;
    const float dyy = D(cl, cx, cy + 1) + D(cl, cx, cy - 1) - 2.0f * c;
    const float dxy =
        0.25f * (D(cl, cx + 1, cy + 1) - D(cl, cx - 1, cy + 1) - D(cl, cx + 1, cy - 1) + D(cl, cx - 1, cy - 1));
#undef D
    const float tr = dxx + dyy;
    const float det = dxx * dyy - dxy * dxy;
    if (det <= 0.0f || tr * tr / det >= a.edge_thr) return;
    const float rs = (float)cl + d[2];
    const uint32_t slot = atomicAdd(a.count, 1u);
    if (slot >= a.cap) return;  // the host sees count > cap and runs again with room
    FeatCand fc;
    fc.x = (float)cx + d[0];
    fc.y = (float)cy + d[1];
    fc.sig = rs;  // candidate_sigma_kernel makes it a scale
    fc.value = value;
    fc.img = (uint16_t)b;
    fc.octave = (uint8_t)a.octave;
    fc.layer = (uint8_t)cl;
    fc.key = ((uint64_t)a.octave << 48) | ((uint64_t)l0 << 32) | ((uint64_t)y << 16) | (uint64_t)x;
    a.cands[slot] = fc;
}

// An octave's gradient tables and its extrema in one launch, the extrema's blocks
// first: neither needs the other, and in small octaves each is a few microseconds
// of latency (one 717 x 531 image with its upsampled detection 1.12 -> 1.05 ms).
static_assert(kGradThreads == 32 * kExtremaWarps, "one block size");
__global__ void __launch_bounds__(kGradThreads) layers_kernel(ExtremaArgs a, int rows, uint3 eg, const float *gauss,
                                                              float2 *grad, uint64_t img_stride, uint3 gg) {
    uint32_t k = grid_wait(blockIdx.x);
    grid_go();
    const uint32_t ne = eg.x * eg.y * eg.z;
    if (k < ne) {  // block-uniform
        extrema_strips(a, rows, make_uint3(k % eg.x, k / eg.x % eg.y, k / (eg.x * eg.y)));
    } else {
        k -= ne;
        grad_tile(gauss, grad, a.w, a.h, a.s, a.layer_stride, img_stride, 1, make_uint3(k % gg.x, k / gg.x % gg.y, k / (gg.x * gg.y)));
    }
}

// sig_oct = sigma0 * kstep^s (features.rs:747) of every candidate, one a thread:
// pow in double is some 300 operations at 2 per clock and SM, which a lone
// lane of the scan paid for by itself.
__global__ void __launch_bounds__(256) candidate_sigma_kernel(FeatCand *cands, const uint32_t *count, uint32_t cap,
                                                              float sigma0, float kstep) {
    grid_wait();
    grid_go();
    const uint32_t n = min(*count, cap);
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256)
        cands[i].sig = sigma0 * (float)pow((double)kstep, (double)cands[i].sig);
}

// --------------------------------------------------------------- orientations

// orientations_with (features.rs:361-420): samples of the (2r+1)^2 window in raster
// order, 32 at a time; lane b owns bins b and b + 32 and adds the samples whose bin
// number's bits (by ballot) are its own, in raster order (0.42 -> 0.19 ms for 24
// views of 960 x 540, against passing all 32 samples to every lane); then the lanes
// smooth and pick the peaks. One warp per candidate, or, while there are fewer
// candidates than the SMs hold CTAs, one CTA: its warps take 32 samples each and
// the first one adds them, set after set (one image's 700 candidates are a warp's
// chain of 50 steps of 0.9 us each: 48 us, 30 with eight warps; with a CTA for each of
// 3000 a call of 24 views takes 2.61 ms instead of 2.39).
constexpr uint32_t kOriFew = 8;  // candidates a SM up to which each has a CTA
struct OriWindow {
    const float2 *grad;
    int w, h, r, xi, yi, side, total;
    float x, y, sw;
};
__device__ __forceinline__ OriWindow ori_window(const OrientArgs &a, uint32_t ci) {
    const FeatCand c = a.cands[ci];
    const OctaveGeom &G = a.geom[c.octave];
    OriWindow W;
    W.grad = a.grads + G.grad_off + ((uint64_t)c.img * a.s + (c.layer - 1)) * G.layer_stride;
    W.w = G.w;
    W.h = G.h;
    W.x = c.x;
    W.y = c.y;
    W.sw = 1.5f * c.sig;
    W.r = f2i(roundf(3.0f * W.sw));
    W.xi = f2i(roundf(c.x));
    W.yi = f2i(roundf(c.y));
    W.side = 2 * W.r + 1;
    W.total = W.side * W.side;
    return W;
}

// Sample t's bin (63: none, no lane's bin) and value.
__device__ __forceinline__ int ori_sample(const OriWindow &W, int t, float &val) {
    val = 0.0f;
    if (t >= W.total) return 63;
    const int px = W.xi + (t % W.side) - W.r, py = W.yi + (t / W.side) - W.r;
    if (px < 1 || py < 1 || px >= W.w - 1 || py >= W.h - 1) return 63;
    const float2 gm = W.grad[(uint64_t)py * W.w + px];
    const float fx = (float)px - W.x, fy = (float)py - W.y;
    const float wgt = exp_cr(-(fx * fx + fy * fy) / (2.0f * W.sw * W.sw));
    const float ang = rem_euclid(gm.y, kTwoPi);
    const float bf = roundf(ang / kTwoPi * (float)kOriBins);
    val = wgt * gm.x;
    return (int)((unsigned)(bf < 0.0f ? 0 : f2i(bf)) % kOriBins);
}

// The lane's bins of 32 samples, whose values lie in vals (by a whole warp).
__device__ __forceinline__ void ori_add(int bin, const float *vals, int lane, float &h0, float &h1) {
    uint32_t low = ~0u;
#pragma unroll
    for (int k = 0; k < 5; ++k)  // the bits that make a bin number this lane's, and (lanes 0-3) this lane's + 32
        low &= __ballot_sync(0xffffffffu, (bin >> k) & 1) ^ ((lane >> k) & 1 ? 0u : ~0u);
    const uint32_t high = __ballot_sync(0xffffffffu, bin >> 5);
    for (uint32_t m = low & ~high; m; m &= m - 1) h0 += vals[__ffs(m) - 1];
    if (lane < kOriBins - 32)
        for (uint32_t m = low & high; m; m &= m - 1) h1 += vals[__ffs(m) - 1];
}

// Smooths the histogram and writes its peaks (by a whole warp).
__device__ __forceinline__ void ori_peaks(const OrientArgs &a, uint32_t ci, float *hist, int lane, float h0, float h1) {
    // six [1,1,1]/3 smoothings, lane b computing bins b and b + 32 (each bin
    // from the previous pass's three, ((l + c) + r) / 3 as the reference)
    const int b1 = lane + 32;
    const bool has1 = b1 < kOriBins;
    for (int it = 0; it < 6; ++it) {
        hist[lane] = h0;
        if (has1) hist[b1] = h1;
        __syncwarp();
        const float n0 = (hist[(lane + kOriBins - 1) % kOriBins] + h0 + hist[(lane + 1) % kOriBins]) / 3.0f;
        const float n1 = has1 ? (hist[(b1 + kOriBins - 1) % kOriBins] + h1 + hist[(b1 + 1) % kOriBins]) / 3.0f : 0.0f;
        __syncwarp();
        h0 = n0;
        h1 = n1;
    }
    hist[lane] = h0;
    if (has1) hist[b1] = h1;
    __syncwarp();
    // fold(0.0, f32::max): fmaxf is order-free (NaN ignored either way)
    float mx = fmaxf(h0, has1 ? h1 : 0.0f);
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mx = fmaxf(0.0f, mx);
    // peaks in bin order: bins 0..31 by lane, then 32..35
    float *out = a.angles + (uint64_t)ci * kMaxAngles;
    int na = 0;
    if (mx > 0.0f) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = half ? b1 : lane;
            bool peak = false;
            float ang = 0.0f;
            if (i < kOriBins) {
                const float l = hist[(i + kOriBins - 1) % kOriBins], cc = hist[i], rr = hist[(i + 1) % kOriBins];
                if (cc >= 0.8f * mx && cc > l && cc > rr) {
                    const float off = 0.5f * (l - rr) / (l - 2.0f * cc + rr);
                    ang = rem_euclid(((float)i + off) / (float)kOriBins * kTwoPi, kTwoPi);
                    peak = true;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, peak);
            if (peak) out[na + __popc(m & ((1u << lane) - 1u))] = ang;
            na += __popc(m);
        }
    }
    if (lane == 0) a.nang[ci] = (uint8_t)na;
}

__global__ void __launch_bounds__(256) orient_kernel(OrientArgs a) {
    __shared__ float hs[8][kOriBins];
    __shared__ float vals[2][8][32];
    __shared__ uint8_t bins[2][8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    grid_wait();
    grid_go();
    const uint32_t n = min(*a.count, a.cap);
    if (n <= a.few) {  // a CTA each
        int par = 0;
        for (uint32_t ci = blockIdx.x; ci < n; ci += gridDim.x) {
            const OriWindow W = ori_window(a, ci);
            float h0 = 0.0f, h1 = 0.0f;
            for (int base = 0; base < W.total; base += 256, par ^= 1) {  // the buffers take turns
                float v;
                bins[par][warp][lane] = (uint8_t)ori_sample(W, base + threadIdx.x, v);
                vals[par][warp][lane] = v;
                __syncthreads();
                if (warp == 0)
                    for (int e = 0; e < 8 && base + 32 * e < W.total; ++e)
                        ori_add(bins[par][e][lane], vals[par][e], lane, h0, h1);
            }
            if (warp == 0) ori_peaks(a, ci, hs[0], lane, h0, h1);
        }
        return;
    }
    for (uint32_t ci = blockIdx.x * 8 + warp; ci < n; ci += gridDim.x * 8) {  // warp-uniform
        const OriWindow W = ori_window(a, ci);
        float h0 = 0.0f, h1 = 0.0f;
        for (int base = 0; base < W.total; base += 32) {
            float v;
            const int bin = ori_sample(W, base + lane, v);
            vals[0][warp][lane] = v;
            __syncwarp();
            ori_add(bin, vals[0][warp], lane, h0, h1);
            __syncwarp();
        }
        ori_peaks(a, ci, hs[warp], lane, h0, h1);
    }
}

// ----------------------------------------------------------------- describe

constexpr int kDescThreads = 128;

// cos and sin of each job's angle, in double rounded to float: one job a
// thread, since FP64 runs at 2 operations per clock and SM (in the describing
// CTAs four warps each repeated them).
__global__ void __launch_bounds__(128) describe_angle_kernel(const DescJob *jobs, float2 *cs, uint32_t n) {
    grid_wait();
    grid_go();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = (double)jobs[i].angle;
    cs[i] = make_float2((float)cos(a), (float)sin(a));
}

// A feature's window: describe_with's scalars (features.rs:521-533).
struct DescWindow {
    const float2 *grad;
    int w, h, xi, yi, r;
    float x, y, c, sn, angle, cell, lim;
    bool geo;  // the rotation is a rotation (false for NaN): rows can be bounded
};

__device__ __forceinline__ DescWindow desc_window(const DescribeArgs &a, uint32_t k, int max_r) {
    const DescJob job = a.jobs[k];
    DescWindow W;
    float sig;
    if (a.cands) {
        const FeatCand c = a.cands[job.cand];
        const OctaveGeom &G = a.geom[c.octave];
        W.grad = a.grads + G.grad_off + ((uint64_t)c.img * a.s + (c.layer - 1)) * G.layer_stride;
        W.w = G.w;
        W.h = G.h;
        W.x = c.x;
        W.y = c.y;
        sig = c.sig;
    } else {  // describe(img, x, y, sigma, angle) on one gradient table
        const slm_keypoint &kp = a.kps[job.cand];
        W.grad = a.grads;
        W.w = a.geom[0].w;
        W.h = a.geom[0].h;
        W.x = kp.x;
        W.y = kp.y;
        sig = kp.sigma;
    }
    const float2 cs = a.cs[k];
    W.c = cs.x;
    W.sn = cs.y;
    W.angle = job.angle;
    W.cell = 3.0f * sig;
    W.r = min(f2i(roundf(W.cell * kSqrt2 * (4.0f + 1.0f) * 0.5f)), max_r);
    W.xi = f2i(roundf(W.x));
    W.yi = f2i(roundf(W.y));
    // |numerator| above 2.6 cells puts bu or bv beyond (-1, 4) whatever the
    // division rounds to: such samples skip the divisions (NaN goes on to the
    // reference's test)
    W.lim = 2.6f * W.cell;
    W.geo = fabsf(W.c) <= 1.0f && fabsf(W.sn) <= 1.0f && W.lim < 1e6f;
    return W;
}

// The samples of window row `row` (0 .. 2r) that can lie inside the rotated
// cells: columns xi + lo .. xi + lo + n - 1, those with |c fx + sn fy| and
// |-sn fx + c fy| within lim widened by a pixel. A superset: the reference's own
// test on each sample decides. (Half of a square window lies outside.)
__device__ __forceinline__ uint32_t desc_row(const DescWindow &W, int row, int &lo) {
    const int py = W.yi + row - W.r;
    lo = max(-W.r, 1 - W.xi);
    int hi = min(W.r, W.w - 2 - W.xi);
    if (py < 1 || py >= W.h - 1) return 0;
    if (W.geo) {
        const float fy = (float)py - W.y, ex = (float)W.xi - W.x;  // fx = dx + ex
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float m = k ? -W.sn : W.c, o = k ? W.c * fy : W.sn * fy;
            if (fabsf(m) < 1e-3f) continue;  // nearly along the row: bounds nothing
            const float e0 = (-W.lim - o) / m - ex, e1 = (W.lim - o) / m - ex;
            lo = max(lo, f2i(floorf(fminf(e0, e1))) - 1);
            hi = min(hi, f2i(ceilf(fmaxf(e0, e1))) + 1);
        }
    }
    return hi >= lo ? hi - lo + 1 : 0;
}

// One sample (features.rs:534-573): false when it lies outside the cells; else
// its weighted magnitude, its place between cells, and its lower cell row + 1, cell
// column + 1 and orientation, 3 bits each.
struct DescSample {
    float m, du, dv, dob;
    uint32_t code;
};
__device__ __forceinline__ bool desc_sample(const DescWindow &W, int px, int py, DescSample &s) {
    const int NC = 4, NO = 8;
    const float fx = (float)px - W.x, fy = (float)py - W.y;
    const float pu = W.c * fx + W.sn * fy, pv_ = -W.sn * fx + W.c * fy;
    if (fabsf(pu) > W.lim || fabsf(pv_) > W.lim) return false;
    const float u = pu / W.cell;
    const float v = pv_ / W.cell;
    const float bu = u + (float)NC / 2.0f - 0.5f, bv = v + (float)NC / 2.0f - 0.5f;
    if (bu <= -1.0f || bv <= -1.0f || bu >= (float)NC || bv >= (float)NC) return false;
    const float2 gm = W.grad[(uint64_t)py * W.w + px];
    const float ori = rem_euclid(gm.y - W.angle, kTwoPi);
    const float bo = ori / kTwoPi * (float)NO;
    const float wgt = exp_cr(-(u * u + v * v) / (2.0f * 4.0f));
    s.m = gm.x * wgt;
    const float u0 = floorf(bu), v0 = floorf(bv), o0 = floorf(bo);
    s.du = bu - u0, s.dv = bv - v0, s.dob = bo - o0;
    const int io0 = o0 < 0.0f ? 0 : f2i(o0);
    s.code = (uint32_t)(f2i(v0) + 1) | (uint32_t)(f2i(u0) + 1) << 3 | (uint32_t)(io0 & (NO - 1)) << 6;
    return true;
}

// Its 8 products m wv wu wo, in the reference's order of factors: k's bits are the
// upper row, column and orientation.
__device__ __forceinline__ void desc_products(const DescSample &s, float (&out)[8]) {
    const float pv[2] = {s.m * (1.0f - s.dv), s.m * s.dv}, wu[2] = {1.0f - s.du, s.du}, wo[2] = {1.0f - s.dob, s.dob};
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = pv[k >> 2] * wu[(k >> 1) & 1] * wo[k & 1];
}

// A warp's samples, SETS times 32 of them, sorted into bins: list holds the
// products of the bins, bin after bin, each bin's in sample order and padded with
// zeros to a multiple of four (adding 0 changes no sum here: none is -0). off and any
// have a border of one cell: a sample's products for rows and columns outside the
// 4 x 4 go to the place after the list.
template <int SETS>
struct __align__(16) DescGroup {
    static constexpr int kMax = 256 * SETS + 3 * 128;  // products, at most 3 zeros a bin
    float list[kMax + 4];
    uint16_t off[6 * 6 * 8];  // first place of bin (row, column, orientation) at ((row + 1) * 6 + column + 1) * 8 + o
    uint32_t any[SETS][6 + 6 + 8];  // samples of a set that touch row -1..4, column -1..4, orientation 0..7
};

template <int SETS>
__device__ __forceinline__ void desc_group_init(DescGroup<SETS> &G, int lane) {
    for (int e = lane; e < 6 * 6 * 8; e += 32) G.off[e] = DescGroup<SETS>::kMax;
    for (int e = lane; e < 20 * SETS; e += 32) G.any[0][e] = 0;
    __syncwarp();
}

// Fills G from each lane's samples, one a set (desc_sample); the sets come one after
// the other in sample order. The bits of the codes by ballot give the mask of the
// samples that touch a row, column or orientation (a lane makes one word); a bin's
// samples are the AND of three, a sample's place in it the number of earlier ones.
// Lane l lays out bins (iv, iu, io), (iv, iu, io + 4), (iv + 2, iu, io) and (iv + 2,
// iu, io + 4) with iv = l / 16, iu = l / 4 % 4, io = l % 4, one after the other: quads
// are their lengths in fours, start the first one's place / 4. Neighbouring samples
// share cells and orientations, so the bins busy at one time lie in different lanes.
template <int SETS>
__device__ __forceinline__ void desc_group(const DescSample (&smp)[SETS], const bool (&valid)[SETS], int lane,
                                           DescGroup<SETS> &G, uint32_t (&quads)[4], uint32_t &start) {
    // the codes of the samples whose lower / upper row, column or orientation this lane's word is for
    const int vu = lane < 8 ? lane & 3 : (lane + 7) & 7, vl = lane < 8 ? (lane & 3) + 1 : lane & 7;
#pragma unroll
    for (int s = 0; s < SETS; ++s) {
        uint32_t b[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) b[k] = __ballot_sync(0xffffffffu, (smp[s].code >> k) & 1u);
        uint32_t lower = __ballot_sync(0xffffffffu, valid[s]), upper = lower;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t t = lane < 4 ? b[k] : lane < 8 ? b[3 + k] : b[6 + k];
            lower &= (vl >> k) & 1 ? t : ~t;
            upper &= (vu >> k) & 1 ? t : ~t;
        }
        if (lane < 16) G.any[s][lane < 4 ? lane + 1 : lane < 8 ? lane + 3 : lane + 4] = lower | upper;
    }
    __syncwarp();
    const int p = lane >> 4, iu = (lane >> 2) & 3, q = lane & 3;
    quads[0] = quads[1] = quads[2] = quads[3] = 3;
#pragma unroll
    for (int s = 0; s < SETS; ++s) {
        const uint32_t *w = G.any[s], c = w[7 + iu], r0 = w[1 + p] & c, r2 = w[3 + p] & c, o0 = w[12 + q], o4 = w[16 + q];
        quads[0] += __popc(r0 & o0);
        quads[1] += __popc(r0 & o4);
        quads[2] += __popc(r2 & o0);
        quads[3] += __popc(r2 & o4);
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) quads[n] >>= 2;
    const uint32_t mine = quads[0] + quads[1] + quads[2] + quads[3];
    uint32_t sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += t;
    }
    start = sum - mine;
    uint16_t *off = &G.off[((p + 1) * 6 + iu + 1) * 8 + q];
    off[0] = (uint16_t)(4 * start);
    off[4] = (uint16_t)(4 * (start + quads[0]));
    off[2 * 48] = (uint16_t)(4 * (start + quads[0] + quads[1]));
    off[2 * 48 + 4] = (uint16_t)(4 * (sum - quads[3]));
    const uint32_t total = __shfl_sync(0xffffffffu, sum, 31);
    for (uint32_t e = lane; e < total; e += 32)
        reinterpret_cast<float4 *>(G.list)[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < SETS; ++s)
        if (valid[s]) {
            float prod[8];
            desc_products(smp[s], prod);
            const uint32_t code = smp[s].code, lt = (1u << lane) - 1;
            const uint32_t v0 = code & 7, u0 = (code >> 3) & 7, o0 = code >> 6, o1 = (o0 + 1) & 7;
            const uint32_t t0 = G.any[s][12 + o0] & lt, t1 = G.any[s][12 + o1] & lt;
            const uint16_t *at = &G.off[(v0 * 6 + u0) * 8];
#pragma unroll
            for (uint32_t d = 0; d < 4; ++d) {  // row v0 - 1 + d / 2, column u0 - 1 + d % 2
                const uint32_t iv = v0 + (d >> 1), iu1 = 6 + u0 + (d & 1);
                const uint32_t m = G.any[s][iv] & G.any[s][iu1];
                const uint16_t *w = at + (d >> 1) * 48 + (d & 1) * 8;
                uint32_t a0 = w[o0] + __popc(m & t0), a1 = w[o1] + __popc(m & t1);
#pragma unroll
                for (int e = 0; e < s; ++e) {  // the earlier sets' samples of the bin
                    const uint32_t me = G.any[e][iv] & G.any[e][iu1];
                    a0 += __popc(me & G.any[e][12 + o0]);
                    a1 += __popc(me & G.any[e][12 + o1]);
                }
                G.list[a0] = prod[2 * d];
                G.list[a1] = prod[2 * d + 1];
            }
        }
}

// n2 of a histogram in index order (features.rs:575-580)
__device__ __forceinline__ float desc_norm(const float *sq) {
    float n2 = -0.0f;
    const float4 *q = reinterpret_cast<const float4 *>(sq);
#pragma unroll 8
    for (int i = 0; i < kDesc / 4; ++i) {
        const float4 f = q[i];
        n2 += f.x;
        n2 += f.y;
        n2 += f.z;
        n2 += f.w;
    }
    return sqrtf(n2);
}

// describe_with (features.rs:521-592). Each of a feature's 128 bins is one f32
// sum over the window's samples in raster order: a serial chain, and on smooth
// images few chains are busy at a time (32 neighbours share cells and nearly an
// orientation: 22 adds in a row for the 136 of a group). So the work around the
// adds is kept small: samples are sorted into bins 64 at a time (desc_group),
// and a bin's owner then runs through its list. (32 at a time, the scan, the
// clearing and the layout are paid twice: 2.49 ms for a call of 24 views, now 2.39,
// and 0.58 for 1500 large windows, now 0.52; with 96 or 128 fewer warps fit: 2.47
// and 2.72.)
//   one warp a feature (windows of up to kDescWarpSide rows: everything the
//   detector makes), four bins a lane. No barriers.
//   one CTA of 8 warps a feature (larger windows, and all when there are few
//   features: the first n_large jobs): the warps sort 64 samples each, then the
//   threads of four of them, one a bin, take their own first group with
//   samples, then the next, so that cells far apart in a row progress together;
//   busy bins are spread over the four warps. (Four warps in all: the 1500
//   keypoints below took 0.76 ms instead of 0.47, the largest window's chain.)
// Bound by instruction issue. Before, with a CTA per feature, each bin walked
// the bits of its samples and formed each product from a 48-byte record: 2.70 ->
// 1.31 ms for the 28.8 K features of 24 views of 960 x 540, 2.4 -> 0.47 ms for
// 1500 keypoints of sigma 1.6 to 13.
constexpr int kDescWarps = kDescThreads / 32;
constexpr int kDescCtaWarps = 8, kDescCtaThreads = 32 * kDescCtaWarps;  // of a large window

constexpr int kDescSets = 2, kDescCtaSets = 2;  // of 32 samples a warp sorts at a time: its own feature's, a CTA's
struct __align__(16) DescWarpSmem {  // one per warp, side by side: list is read as float4
    DescGroup<kDescSets> g;
    uint32_t first[kDescWarpSide + 1];
    int16_t left[kDescWarpSide + 1];
};
static_assert(sizeof(DescWarpSmem) % 16 == 0 && sizeof(DescGroup<kDescCtaSets>) % 16 == 0 && sizeof(DescGroup<kDescSets>) % 16 == 0, "alignment of the vector accesses");
struct __align__(16) DescCtaSmem {
    DescGroup<kDescCtaSets> g[2][kDescCtaWarps];
    uint32_t wsum[kDescCtaWarps];
    float norm;
};

__device__ void describe_warp(const DescribeArgs &a, uint32_t k, DescWarpSmem &S, int lane) {
    const DescWindow W = desc_window(a, k, (kDescWarpSide - 1) / 2);
    const int side = 2 * W.r + 1;
    uint32_t total = 0;
    for (int base = 0; base < side; base += 32) {
        const int row = base + lane;
        int lo = 0;
        const uint32_t n = row < side ? desc_row(W, row, lo) : 0;
        uint32_t s = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (row < side) {
            S.first[row] = total + s - n;
            S.left[row] = (int16_t)lo;
        }
        total += __shfl_sync(0xffffffffu, s, 31);
    }
    if (lane == 0) S.first[side] = total;
    __syncwarp();
    desc_group_init(S.g, lane);
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // this lane's bins (desc_group)
    int row = 0;
    for (uint32_t base = 0; base < total; base += 32 * kDescSets) {
        DescSample smp[kDescSets];
        bool valid[kDescSets];
        uint32_t n[4], at;
#pragma unroll
        for (int e = 0; e < kDescSets; ++e) {
            const uint32_t t = base + 32 * e + lane;
            valid[e] = false;
            smp[e].code = 0;
            if (t < total) {
                while (t >= S.first[row + 1]) ++row;
                const int px = W.xi + S.left[row] + (int)(t - S.first[row]), py = W.yi + row - W.r;
                valid[e] = desc_sample(W, px, py, smp[e]);
            }
        }
        desc_group<kDescSets>(smp, valid, lane, S.g, n, at);
        __syncwarp();
        // the lane's bins lie one after the other; each run of four is one bin's
        const float4 *l = reinterpret_cast<const float4 *>(S.g.list) + at;
        const uint32_t e1 = n[0], e2 = e1 + n[1], e3 = e2 + n[2], e4 = e3 + n[3];
        for (uint32_t i = 0; i < e4; ++i) {
            const float4 f = l[i];
            const bool b0 = i < e1, b1 = i < e2, b2 = i < e3;
            float s = b0 ? acc[0] : b1 ? acc[1] : b2 ? acc[2] : acc[3];
            s += f.x;
            s += f.y;
            s += f.z;
            s += f.w;
            acc[0] = b0 ? s : acc[0];
            acc[1] = b1 && !b0 ? s : acc[1];
            acc[2] = b2 && !b1 ? s : acc[2];
            acc[3] = b2 ? acc[3] : s;
        }
        __syncwarp();
    }
    const int p = lane >> 4, iu = (lane >> 2) & 3, q = lane & 3;  // bin n: row p + (n & 2), orientation q + 4 (n & 1)
    // normalise, clip, normalise (features.rs:575-590); the histogram goes through the list's space
    float *hist = S.g.list;
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int n = 0; n < 4; ++n) hist[((p + (n & 2)) * 4 + iu) * 8 + q + (n & 1) * 4] = acc[n] * acc[n];
        __syncwarp();
        float nrm = lane == 0 ? desc_norm(hist) : 0.0f;
        nrm = __shfl_sync(0xffffffffu, nrm, 0);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            if (nrm > 0.0f) acc[n] = acc[n] / nrm;
            if (pass == 0) acc[n] = fminf(acc[n], 0.2f);
        }
        __syncwarp();
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) hist[((p + (n & 2)) * 4 + iu) * 8 + q + (n & 1) * 4] = acc[n];
    __syncwarp();
    reinterpret_cast<float4 *>(a.desc + (uint64_t)a.jobs[k].out_row * kDesc)[lane] = reinterpret_cast<float4 *>(hist)[lane];
    __syncwarp();
}

__device__ void describe_cta(const DescribeArgs &a, uint32_t k, DescCtaSmem &S, uint32_t *first) {
    int16_t *left = reinterpret_cast<int16_t *>(first + a.max_side + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const DescWindow W = desc_window(a, k, (a.max_side - 1) / 2);
    const int side = 2 * W.r + 1;
    uint32_t total = 0;
    for (int base = 0; base < side; base += kDescCtaThreads) {
        const int row = base + tid;
        int lo = 0;
        const uint32_t n = row < side ? desc_row(W, row, lo) : 0;
        uint32_t s = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (lane == 31) S.wsum[warp] = s;
        __syncthreads();
        uint32_t all = 0, mine = total + s - n;
#pragma unroll
        for (int g = 0; g < kDescCtaWarps; ++g) {
            if (g < warp) mine += S.wsum[g];
            all += S.wsum[g];
        }
        if (row < side) {
            first[row] = mine;
            left[row] = (int16_t)lo;
        }
        total += all;
        __syncthreads();
    }
    if (tid == 0) first[side] = total;
    __syncthreads();
    const bool owner = warp < 4;
    desc_group_init(S.g[0][warp], lane);
    desc_group_init(S.g[1][warp], lane);
    // bins: one a thread of warps 0-3, busy ones (neighbouring rows and
    // orientations) in different warps
    const int iv = (lane >> 4) * 2 + ((warp >> 1) & 1), iu = (lane >> 2) & 3, io = (lane & 3) * 2 + (warp & 1);
    const uint32_t place = ((iv + 1) * 6 + iu + 1) * 8 + io;
    float acc = 0.0f;  // bin (iv, iu, io)
    int row = 0, par = 0;
    for (uint32_t base = 0; base < total; base += kDescCtaThreads * kDescCtaSets, par ^= 1) {
        uint32_t n[4], at;
        DescSample smp[kDescCtaSets];
        bool valid[kDescCtaSets];
#pragma unroll
        for (int e = 0; e < kDescCtaSets; ++e) {
            const uint32_t t = base + 32 * (kDescCtaSets * warp + e) + lane;
            valid[e] = false;
            smp[e].code = 0;
            if (t < total) {
                while (t >= first[row + 1]) ++row;
                const int px = W.xi + left[row] + (int)(t - first[row]), py = W.yi + row - W.r;
                valid[e] = desc_sample(W, px, py, smp[e]);
            }
        }
        desc_group<kDescCtaSets>(smp, valid, lane, S.g[par][warp], n, at);
        __syncthreads();  // one for the warps' samples: the buffers take turns
        if (!owner) continue;
        uint32_t some = 0;
#pragma unroll
        for (int g = 0; g < kDescCtaWarps; ++g) {
            const DescGroup<kDescCtaSets> &G = S.g[par][g];
            uint32_t m = 0;
#pragma unroll
            for (int e = 0; e < kDescCtaSets; ++e) m |= G.any[e][1 + iv] & G.any[e][7 + iu] & G.any[e][12 + io];
            some |= m ? 1u << g : 0u;
        }
        while (some) {
            const DescGroup<kDescCtaSets> &G = S.g[par][__ffs(some) - 1];
            some &= some - 1;
            const float4 *l = reinterpret_cast<const float4 *>(G.list + G.off[place]);
            int m = 0;
#pragma unroll
            for (int e = 0; e < kDescCtaSets; ++e) m += __popc(G.any[e][1 + iv] & G.any[e][7 + iu] & G.any[e][12 + io]);
            for (int i = 0; i < m; i += 4, ++l) {
                const float4 f = *l;
                acc += f.x;
                acc += f.y;
                acc += f.z;
                acc += f.w;
            }
        }
    }
    const int bin = (iv * 4 + iu) * 8 + io;
    __syncthreads();
    float *sq = S.g[0][0].list;
    float v = acc;
    for (int pass = 0; pass < 2; ++pass) {
        if (owner) sq[bin] = v * v;
        __syncthreads();
        if (tid == 0) S.norm = desc_norm(sq);
        __syncthreads();
        const float nrm = S.norm;
        if (nrm > 0.0f) v = v / nrm;
        if (pass == 0) v = fminf(v, 0.2f);
    }
    if (owner) a.desc[(uint64_t)a.jobs[k].out_row * kDesc + bin] = v;
}

union DescMixedSmem {  // followed by a large window's rows: 4 (max_side + 1) + 2 max_side bytes
    DescWarpSmem warp[kDescCtaWarps];
    DescCtaSmem cta;
};
// Rows of the largest window a detector configuration can ask for: its base
// blur takes sigma0 up to 42.4, a candidate's scale is at most 2^1.5 of that.
constexpr int kDescMaxSide = 2600;

// Blocks 0 .. n_large - 1: a large window each; the rest: eight jobs each. One
// launch for both, so that small windows fill the GPU beside the last large ones.
__global__ void __launch_bounds__(kDescCtaThreads) describe_mixed_kernel(DescribeArgs a, uint32_t njobs) {
    extern __shared__ __align__(16) unsigned char desc_smem[];
    DescMixedSmem &S = *reinterpret_cast<DescMixedSmem *>(desc_smem);
    grid_wait();
    if (blockIdx.x < a.n_large) {
        describe_cta(a, blockIdx.x, S.cta, reinterpret_cast<uint32_t *>(desc_smem + sizeof(DescMixedSmem)));
        return;
    }
    const uint32_t k = a.n_large + (blockIdx.x - a.n_large) * kDescCtaWarps + (threadIdx.x >> 5);
    if (k < njobs) describe_warp(a, k, S.warp[threadIdx.x >> 5], threadIdx.x & 31);
}

// Without large windows (the detector's features): less shared memory and
// fewer registers a CTA.
__global__ void __launch_bounds__(kDescThreads, 8) describe_kernel(DescribeArgs a, uint32_t njobs) {
    __shared__ DescWarpSmem S[kDescWarps];
    grid_wait();
    const uint32_t k = blockIdx.x * kDescWarps + (threadIdx.x >> 5);
    if (k < njobs) describe_warp(a, k, S[threadIdx.x >> 5], threadIdx.x & 31);
}

}  // namespace

namespace {
struct BlurFused {
    void (*kernel)(const float *, float *, float *, int, int, uint64_t, uint64_t, uint64_t, BlurTaps);
    size_t smem;
    int rows;  // output rows of a tile
};
// The fused kernel of radius r (1 .. kFusedR).
template <int R>
BlurFused blur_of_radius(int r, bool tall) {
    if constexpr (R < kFusedR)
        if (r > R) return blur_of_radius<R + 1>(r, tall);
    if (tall) return {blur_fused_kernel<R, true>, blur_smem<R, true>(), blur_rows<R, true>()};
    return {blur_fused_kernel<R, false>, blur_smem<R, false>(), blur_rows<R, false>()};
}
}  // namespace

cudaError_t init_feature_kernels() {
    for (int r = 1; r <= kFusedR; ++r)
        for (int tall = 0; tall < 2; ++tall) {
            const BlurFused f = blur_of_radius<1>(r, tall != 0);
            const cudaError_t e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.smem);
            if (e != cudaSuccess) return e;
        }
    return cudaFuncSetAttribute(describe_mixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(DescMixedSmem) + 6 * (kDescMaxSide + 1)));
}

void launch_blur(const float *src, float *tmp, float *dst, const float *prev, float *dog, int w, int h, int nimg,
                 uint64_t stride_src, uint64_t stride_dst, uint64_t stride_dog, const BlurTaps &t, int sms, cudaStream_t s) {
    if (t.r <= kFusedR && (!dog || (prev == src && stride_src == stride_dst))) {
        // tall tiles (less halo) once they still give every SM four: 0.61 -> 0.58 ms for
        // 24 views of 960 x 540 in one launch, where one photo's would leave SMs idle (a
        // batch's parts have fewer tiles: the large images of a call are what takes them)
        const uint64_t tiles = (uint64_t)((w + kFX - 1) / kFX) * ((h + 63) / 64) * nimg;
        const BlurFused f = blur_of_radius<1>(t.r, tiles >= 4ull * sms);
        const dim3 g((w + kFX - 1) / kFX, (h + f.rows - 1) / f.rows, nimg);
        launch_next(f.kernel, g, 256, f.smem, s, src, dst, dog, w, h, stride_src, stride_dst, stride_dog, t);
        return;
    }
    const dim3 grid((w + kBlurX - 1) / kBlurX, h, nimg);
    launch_next(blur_rows_kernel, grid, kBlurX, 0, s, src, tmp, w, h, stride_src, (uint64_t)w * h, t);
    launch_next(blur_cols_kernel, grid, kBlurX, 0, s, tmp, dst, prev, dog, w, h, (uint64_t)w * h, stride_dst, stride_dog, t);
}

void launch_downsample(const float *src, float *dst, int w, int h, int nimg, uint64_t stride_src,
                       uint64_t stride_dst, cudaStream_t s) {
    const int nw = w / 2, nh = h / 2;
    if (!nw || !nh) return;
    launch_next(downsample_kernel, dim3((nw + 255) / 256, nh, nimg), 256, 0, s, src, dst, w, h, nw, nh, stride_src,
                stride_dst);
}

void launch_upsample2(const float *src, float *dst, int w, int h, int nimg, cudaStream_t s) {
    launch_next(upsample2_kernel, dim3((2 * w + 255) / 256, 2 * h, nimg), 256, 0, s, src, dst, w, h);
}

void launch_gray_from_rgb8(const uint8_t *rgb, float *out, uint64_t n, cudaStream_t s) {
    if (n)
        launch_next(gray_from_rgb8_kernel, (unsigned)((n + 1023) / 1024), 256, 0, s, rgb, out, n,
                    (reinterpret_cast<uintptr_t>(rgb) & 3) == 0);
}

void launch_read_images(const float *src, float *dst, uint64_t n, int sms, cudaStream_t s) {
    const uint64_t n4 = n / 4;
    if (n4)
        launch_next(read_images_kernel, (unsigned)((n4 + 255) / 256 < 8ull * sms ? (n4 + 255) / 256 : 8ull * sms), 256, 0, s,
                    reinterpret_cast<const float4 *>(src), reinterpret_cast<float4 *>(dst), n4);
}

void launch_grad(const float *gauss, float2 *grad, int w, int h, int s_, uint64_t img_stride, int l0, int nimg,
                 cudaStream_t s) {
    launch_next(grad_kernel, dim3((w + kGradThreads - 1) / kGradThreads, (h + kGradRows - 1) / kGradRows, nimg * s_),
                kGradThreads, 0, s, gauss, grad, w, h, s_, (uint64_t)w * h, img_stride, l0);
}

void launch_layers(const ExtremaArgs &a, const float *gauss, float2 *grad, uint64_t img_stride, int nimg, int sms,
                   cudaStream_t s) {
    // strips of 16 rows where that leaves every SM its 16 warps, else of 4
    const uint64_t warps = (uint64_t)((a.w + 27) / 30) * ((a.h + 13) / 16) * nimg * a.s;
    const int rows = warps >= 16ull * sms ? kExtremaRows : 4, strip = kExtremaWarps * rows;
    const uint32_t layers = (uint32_t)nimg * a.s;
    const uint3 gg = make_uint3((a.w + kGradThreads - 1) / kGradThreads, (a.h + kGradRows - 1) / kGradRows, layers);
    const uint3 eg = a.w < 3 || a.h < 3 ? make_uint3(1, 1, 0)
                                        : make_uint3((a.w + 27) / 30, (a.h - 2 + strip - 1) / strip, layers);
    launch_next(layers_kernel, eg.x * eg.y * eg.z + gg.x * gg.y * gg.z, kGradThreads, 0, s, a, rows, eg, gauss, grad,
                img_stride, gg);
}

// The number of candidates is the device's: grids for as many as there may be,
// up to what the SMs hold a few times over.
void launch_candidate_sigma(FeatCand *cands, const uint32_t *count, uint32_t cap, float sigma0, float kstep, int sms,
                            cudaStream_t s) {
    const uint32_t grid = (cap + 255) / 256 < 2u * sms ? (cap + 255) / 256 : 2u * sms;
    launch_next(candidate_sigma_kernel, grid, 256, 0, s, cands, count, cap, sigma0, kstep);
}

void launch_orient(const OrientArgs &a, int sms, cudaStream_t s) {
    const uint32_t grid = (a.cap + 7) / 8 < 16u * sms ? (a.cap + 7) / 8 : 16u * sms;
    OrientArgs b = a;
    b.few = kOriFew * (uint32_t)sms;
    launch_next(orient_kernel, grid, 256, 0, s, b);
}

void launch_describe(const DescribeArgs &a, uint32_t njobs, cudaStream_t s) {
    if (!njobs) return;
    launch_next(describe_angle_kernel, (njobs + 127) / 128, 128, 0, s, a.jobs, a.cs, njobs);
    if (!a.n_large) {
        launch_next(describe_kernel, (njobs + kDescWarps - 1) / kDescWarps, kDescThreads, 0, s, a, njobs);
        return;
    }
    const size_t rows = sizeof(DescMixedSmem) + 4 * (size_t)(a.max_side + 1) + 2 * (size_t)a.max_side;
    launch_next(describe_mixed_kernel, a.n_large + (njobs - a.n_large + kDescCtaWarps - 1) / kDescCtaWarps, kDescCtaThreads,
                rows, s, a, njobs);
}

}  // namespace slm
