// k_sampson.cu — batched Sampson scoring of essential-matrix hypotheses.
//
// Reference: crates/core/src/two_view.rs:456-465 (`sampson_residual`) and
// :804-823 (`inliers_of` and `count_at_least` in ransac_essential_inner, the
// per-hypothesis work of the RANSAC stage that runs on every pair kept by
// match_pairs, pipeline.rs:505). The reference scores each 5-point hypothesis
// over the pair's matches in f64; here one warp scores one hypothesis, 32
// matches at a time, every residual in the reference's f64 operation order
// (explicit round-to-nearest operations: nothing is contracted to an FMA), so
// counts and inlier sets are the reference's bit for bit. count_at_least's
// early exit changes only when it stops, not its answer: it returns the full
// count when that reaches `need` and nothing otherwise, so the full count
// settles it.
//
// What bounds it: FP64. A residual is about 70 f64 operations at 2 per clock
// and SM; all of them in f64 took 8.1 ms for 77 M residuals (100 pairs, 2000
// hypotheses each). So a match is first tested in FP32 with an error bound:
// the test |dot| < th * den holds or fails for certain unless the two sides
// come within the bound (a few matches in 10^5 of a wrong hypothesis, a few in
// 10^3 of a near-true one), and only then is the f64 residual formed. The
// counts and masks stay the f64 residual's, since a certain answer is its
// answer whatever the roundings. The same call from host arrays, with 100 masks
// read back as Python arrays, went from 8.8 to 0.82 ms; the C call without them takes
// 0.40 of it, the 14 MB of hypotheses read over the link where they lie. A
// hypothesis beyond the FP32 test's range is f64 throughout and reads its
// entries again, through the cache, for every 32 matches: a call of nothing
// else takes 8.4 ms. (Its entries kept in shared memory: no faster, and the
// usual call slower.)
#include <cuda_runtime.h>

#include <cstdint>

#include "slm_internal.h"

namespace slm {

namespace {

// The signed residual e p . q / |grad| of one correspondence, p = (ax, ay, 1),
// q = (bx, by, 1), e row-major. The order is the reference's linear algebra:
// row i of e p is ((e[i][0] ax + e[i][1] ay) + e[i][2] 1), the same for
// e^T q with the rows of e^T; den = sqrt(((ep0^2 + ep1^2) + etq0^2) + etq1^2);
// the residual is (bx ep0 + by ep1 + ep2) / den, or 0 when den is not > 0
// (also when it is NaN). Division and square root are IEEE round-to-nearest.
__device__ __forceinline__ double residual(const double (&e)[9], double ax, double ay, double bx, double by) {
    double ep[3], etq[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double y = __dmul_rn(e[3 * i], ax);
        y = __dadd_rn(__dmul_rn(e[3 * i + 1], ay), y);
        ep[i] = __dadd_rn(__dmul_rn(e[3 * i + 2], 1.0), y);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double y = __dmul_rn(e[i], bx);
        y = __dadd_rn(__dmul_rn(e[3 + i], by), y);
        etq[i] = __dadd_rn(__dmul_rn(e[6 + i], 1.0), y);
    }
    const double s = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(ep[0], ep[0]), __dmul_rn(ep[1], ep[1])),
                                         __dmul_rn(etq[0], etq[0])),
                               __dmul_rn(etq[1], etq[1]));
    const double den = __dsqrt_rn(s);
    if (den > 0.0) {
        const double dot = __dadd_rn(__dadd_rn(__dmul_rn(bx, ep[0]), __dmul_rn(by, ep[1])), __dmul_rn(1.0, ep[2]));
        return __ddiv_rn(dot, den);
    }
    return 0.0;
}

constexpr int kWarpsPerBlock = 8;

// Whether |r| < th, decided in FP32 where that is certain: 1 yes, 0 no, -1 not
// decided. e is the hypothesis scaled by a power of two to a largest entry in
// [1/2, 1) (the residual does not change), q the match, both rounded to f32,
// th in [2^-60, 2^60]. With u = 2^-24, P = |ax| + |ay| + 1 and Q likewise of b:
//   each component of e p is within 4.01 u P of its real value (two rounded
//   inputs, two fused roundings), each of e^T q within 4.01 u Q, the dot product
//   within 8 u P Q, and den, a Euclidean norm of four of them, within
//   6 u (P + Q) + 5 u den (its sum, sqrt.approx at 2^-23).
// The constants below also cover the roundings of the test itself and those of
// the f64 residual (2^-53 relative to the same magnitudes). den must be
// certainly positive for a "no": the residual of a zero den is 0, an inlier.
// NaN and coordinates above 2^60 decide nothing.
__device__ __forceinline__ int certain_inlier(const float (&e)[9], const float4 q, float th) {
    constexpr float u = 0x1p-24f;
    const float P = fabsf(q.x) + fabsf(q.y) + 1.0f, Q = fabsf(q.z) + fabsf(q.w) + 1.0f;
    const float ep0 = fmaf(e[0], q.x, fmaf(e[1], q.y, e[2]));
    const float ep1 = fmaf(e[3], q.x, fmaf(e[4], q.y, e[5]));
    const float ep2 = fmaf(e[6], q.x, fmaf(e[7], q.y, e[8]));
    const float et0 = fmaf(e[0], q.z, fmaf(e[3], q.w, e[6]));
    const float et1 = fmaf(e[1], q.z, fmaf(e[4], q.w, e[7]));
    const float dot = fabsf(fmaf(q.z, ep0, fmaf(q.w, ep1, ep2)));
    float den;
    asm("sqrt.approx.f32 %0, %1;"
        : "=f"(den)
        : "f"(fmaf(ep0, ep0, fmaf(ep1, ep1, fmaf(et0, et0, et1 * et1)))));
    const float PQ = P * Q, ed = 12.0f * u * PQ, eg = 7.0f * u * (P + Q);
    const float lo = fmaf(den, 1.0f - 16.0f * u, -eg), hi = fmaf(den, 1.0f + 16.0f * u, eg);
    if (!(PQ < 0x1p60f)) return -1;
    if (dot + ed < th * lo) return 1;
    if (lo > 0.0f && dot - ed >= th * hi) return 0;
    return -1;
}

// The matches rounded to f32, once a call: a conversion in the scoring loop
// would go through the FP64 pipe for every hypothesis.
__global__ void __launch_bounds__(256) sampson_round_kernel(const double4 *pts, float4 *pts32, uint64_t m) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double4 q = pts[i];
    pts32[i] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
}

// One warp per hypothesis: its pair's matches 32 at a time, the inlier bits
// of each group of 32 by ballot (one mask word, written by lane 0 when the
// hypothesis asks for its mask), the count by population count. A hypothesis
// whose entries or threshold leave the range of the FP32 test (2^-200..2^200
// for the largest entry) is scored in f64 throughout.
__global__ void __launch_bounds__(32 * kWarpsPerBlock) sampson_kernel(SampsonArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t h = (uint64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (h >= a.nh) return;  // warp-uniform
    const uint32_t p = a.hyp_pair[h];
    const uint64_t m0 = a.pair_off[p], m1 = a.pair_off[p + 1];
    const double th = a.thresh[p];
    // lane k < 9 holds entry k; the scaling moves its exponent field
    const long long bits = lane < 9 ? __double_as_longlong(a.E[9 * h + lane]) : 0;
    const int ex = (int)((bits >> 52) & 0x7ff);
    const int top = __reduce_max_sync(0xffffffffu, ex);
    const bool fast = top >= 1023 - 200 && top <= 1023 + 200 && th >= 0x1p-60 && th <= 0x1p60;
    const int scaled = ex + (1022 - top);  // entries below 2^-900 of the largest become 0
    const float mine = ex > 0 && scaled > 0 && fast
                           ? (float)__longlong_as_double((bits & ~(0x7ffll << 52)) | ((long long)scaled << 52))
                           : 0.0f;
    float e32[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) e32[k] = __shfl_sync(0xffffffffu, mine, k);
    const float th32 = (float)th;
    uint32_t *mk = nullptr;
    if (a.masks && a.mask_off && a.mask_off[h] != ~0ull) mk = a.masks + a.mask_off[h];
    uint32_t c = 0;
    for (uint64_t i0 = m0; i0 < m1; i0 += 32) {
        const uint64_t i = i0 + lane;
        int in = 0;
        if (i < m1) {
            in = fast ? certain_inlier(e32, a.pts32[i], th32) : -1;
            if (in < 0) {
                double e[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) e[k] = a.E[9 * h + k];
                const double4 q = a.pts[i];
                // inliers_of / count_at_least: |r| < th, strict (two_view.rs:806, :812)
                in = fabs(residual(e, q.x, q.y, q.z, q.w)) < th;
            }
        }
        const uint32_t word = __ballot_sync(0xffffffffu, in > 0);
        c += __popc(word);
        if (mk && lane == 0) mk[(i0 - m0) >> 5] = word;
    }
    if (lane == 0) a.counts[h] = c;
}

}  // namespace

void launch_sampson(const SampsonArgs &a, cudaStream_t s) {
    if (!a.nh) return;
    if (a.n_pts) sampson_round_kernel<<<(unsigned)((a.n_pts + 255) / 256), 256, 0, s>>>(a.pts, a.pts32, a.n_pts);
    const uint64_t blocks = (a.nh + kWarpsPerBlock - 1) / kWarpsPerBlock;
    sampson_kernel<<<(unsigned)blocks, 32 * kWarpsPerBlock, 0, s>>>(a);
}

}  // namespace slm
