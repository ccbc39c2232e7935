// A CUDA runtime and kernel launchers that run nothing, so that the library's host
// code (csrc/slm.cpp, included by host_checks.cpp) can be checked without a GPU:
// device memory is host memory, copies are made at once, kernels do nothing but leave
// their arguments here. A check can make a call fail, and reads what was called from
// the log.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "slm_internal.h"
#include "slm_shortlist.h"

namespace fake {
inline std::mutex mu;
inline std::vector<std::string> log;        // what was called, in order
inline std::map<void *, size_t> device;     // live device allocations
inline size_t device_bytes = 0, device_peak = 0;
inline int fail_d2h = 0;                    // the n-th copy to the host from now on fails (0: none)
inline slm::TrackArgs tracks{};
inline slm::SampsonArgs sampson{};
inline slm::SlArgs shortlist{};
inline slm::ExactArgs exact{};
inline std::vector<slm::DescribeArgs> describes;

inline void note(const char *what) {
    std::lock_guard<std::mutex> g(mu);
    log.emplace_back(what);
}
inline cudaError_t alloc(void **p, size_t n) {
    std::lock_guard<std::mutex> g(mu);
    *p = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);  // zeros
    if (*p == MAP_FAILED) return *p = nullptr, cudaErrorMemoryAllocation;
    device[*p] = n;
    device_bytes += n;
    if (device_bytes > device_peak) device_peak = device_bytes;
    return cudaSuccess;
}
inline cudaError_t release(void *p) {
    std::lock_guard<std::mutex> g(mu);
    auto it = device.find(p);
    if (it == device.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    device_bytes -= it->second;
    munmap(p, it->second ? it->second : 1);
    device.erase(it);
    return cudaSuccess;
}
inline bool on_device(const void *p) {
    std::lock_guard<std::mutex> g(mu);
    auto it = device.upper_bound(const_cast<void *>(p));
    if (it == device.begin()) return false;
    --it;
    return static_cast<const char *>(p) < static_cast<char *>(it->first) + it->second;
}
inline cudaError_t copy(void *d, const void *s, size_t n) {
    if (on_device(s) && !on_device(d)) {
        std::lock_guard<std::mutex> g(mu);
        if (fail_d2h && --fail_d2h == 0) {
            log.emplace_back("copy failed");
            return cudaErrorUnknown;
        }
    }
    std::memcpy(d, s, n);
    return cudaSuccess;
}
template <class T>
T handle() {
    static std::uintptr_t next = 0x1000;
    std::lock_guard<std::mutex> g(mu);
    return reinterpret_cast<T>(next += 16);
}
}  // namespace fake

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10, p->minor = 3, p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 1, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = size_t(280) << 30, cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaFree(void *p) { return fake::release(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { return *p = fake::handle<cudaMemPool_t>(), cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return fake::alloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return fake::release(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = std::calloc(n ? n : 1, 1), cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return *p = std::calloc(n ? n : 1, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::memset(a, 0, sizeof *a);
    a->type = fake::on_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return fake::copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { return fake::copy(d, s, n); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = fake::handle<cudaStream_t>(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return fake::note("sync"), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) { return *c = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = fake::handle<cudaGraph_t>(), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return *e = fake::handle<cudaGraphExec_t>(), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return fake::note("graph"), cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = fake::handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = fake::handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
}

namespace slm {
cudaError_t init_exact_kernels() { return cudaSuccess; }
cudaError_t init_shortlist_kernels() { return cudaSuccess; }
cudaError_t init_top2_kernels() { return cudaSuccess; }
cudaError_t init_feature_kernels() { return cudaSuccess; }
void launch_exact(const ExactArgs &a, int, cudaStream_t) { fake::exact = a; }
void launch_finalize(const FinalizeArgs &, cudaStream_t) {}
void launch_wait_selftest(uint32_t, uint32_t *, cudaStream_t) {}
void launch_fill_u64(unsigned long long *, uint64_t, unsigned long long, cudaStream_t) {}
void launch_fill_u32(uint32_t *, uint64_t, uint32_t, cudaStream_t) {}
void launch_pack_fp32_tiles(const uint4 *, uint32_t, const float *, float *, cudaStream_t) {}
void launch_pack_lowp(const uint4 *, uint32_t, const float *, int, uint8_t *, float *, float *, ViewStat *, cudaStream_t) {}
void launch_gather(const uint2 *, const uint64_t *, const uint32_t *, const uint64_t *, uint32_t, uint2 *, uint64_t, cudaStream_t) {}
void launch_copy_pairs(const uint2 *, const uint64_t *, slm_pair *, uint32_t, uint32_t *, cudaStream_t) {}
void launch_gather_rows(const uint4 *, uint32_t, float *, cudaStream_t) { fake::note("gather rows"); }
void launch_scatter_rows(const uint4 *, uint32_t, const float *, float *, cudaStream_t) {}
void launch_scan_counts(const uint32_t *, uint32_t, uint64_t *, cudaStream_t) {}
void launch_filter_counts(uint32_t *, uint32_t, uint32_t, cudaStream_t) {}
void launch_gather_blocks(const SlArgs &, const uint64_t *, const uint64_t *, uint2 *, uint64_t, cudaStream_t) {}
SingleLayout single_layout(uint32_t, uint32_t, int, bool) { return SingleLayout{}; }
cudaError_t single_exact_enqueue(unsigned char *, const SingleLayout &, const float *, uint32_t, const float *, uint32_t, float, int,
                                 slm_pair *, uint32_t, uint32_t *, int, cudaStream_t) { return cudaSuccess; }
int launch_shortlist_eps(const SlArgs &a, cudaStream_t) { return fake::shortlist = a, 1; }
int launch_top2_pass(const SlArgs &, cudaStream_t) { return 1; }
int launch_top2_decide(const SlArgs &, int, cudaStream_t) { return 1; }
int launch_top2_resolve(const SlArgs &, int, cudaStream_t) { return 1; }
int launch_shortlist_pass(const SlArgs &, int, int, cudaStream_t) { return 1; }
int launch_shortlist_sample(const SlArgs &, int, cudaStream_t) { return 1; }
int launch_shortlist_mid(const SlArgs &, cudaStream_t) { return 1; }
int launch_shortlist_finalize(const SlArgs &, cudaStream_t) { return 1; }
int launch_shortlist_rescue_prep(const SlArgs &, cudaStream_t) { return 1; }
int launch_shortlist_tail(const SlArgs &, int, cudaStream_t) { return 1; }
void launch_sampson(const SampsonArgs &a, cudaStream_t) { fake::note("sampson"), fake::sampson = a; }
void launch_blur(const float *, float *, float *, const float *, float *, int, int, int, uint64_t, uint64_t, uint64_t, const BlurTaps &, int, cudaStream_t) {}
void launch_grad(const float *, float2 *, int, int, int, uint64_t, int, int, cudaStream_t) {}
void launch_layers(const ExtremaArgs &, const float *, float2 *, uint64_t, int, int, cudaStream_t) {}
void launch_orient(const OrientArgs &, int, cudaStream_t) {}
void launch_describe(const DescribeArgs &a, uint32_t, cudaStream_t) { fake::describes.push_back(a); }
void launch_upsample2(const float *, float *, int, int, int, cudaStream_t) {}
void launch_downsample(const float *, float *, int, int, int, uint64_t, uint64_t, cudaStream_t) {}
void launch_read_images(const float *, float *, uint64_t, int, cudaStream_t) {}
void launch_gray_from_rgb8(const uint8_t *, float *, uint64_t, cudaStream_t) {}
void launch_candidate_sigma(FeatCand *, const uint32_t *, uint32_t, float, float, int, cudaStream_t) {}
void launch_tracks(const TrackArgs &a, uint32_t, int, cudaStream_t) { fake::note("tracks"), fake::tracks = a; }
}  // namespace slm
