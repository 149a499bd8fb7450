// The CUDA runtime and the kernel launchers behind pa_engine.cu, faked on the host: every call that touches a stream is
// logged, allocations are counted, and a named call can be made to fail.
#include "pa_kernels.cuh"

#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

struct pa_engine;

namespace {
std::string log_text, fail_name;
int fail_skip = 0;            // calls of fail_name that still succeed
size_t held = 0, limit = ~size_t(0);
float residual = 0.f;         // what an FP32 block leaves
std::map<void*, size_t> sizes;

// Whether the call `name` fails now.
bool fails(const char* name) {
    log_text += name;
    log_text += '\n';
    return fail_name == name && fail_skip-- <= 0;
}
cudaError_t status(const char* name) { return fails(name) ? cudaErrorUnknown : cudaSuccess; }
// Large buffers are addresses only.
cudaError_t allocate(void** p, size_t n) {
    if (held + n > limit) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, n > (size_t(64) << 20) ? 64 : n);
    sizes[*p] = n;
    held += n;
    return cudaSuccess;
}
cudaError_t release(void* p) {
    if (p) held -= sizes[p];
    sizes.erase(p);
    std::free(p);
    return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_reset() {
    log_text.clear();
    fail_name.clear();
    limit = ~size_t(0);
    residual = 0.f;
}
void fake_fail(const char* name, int skip) {
    fail_name = name;
    fail_skip = skip;
}
void fake_residual(float r) { residual = r; }
void fake_limit(size_t bytes) { limit = bytes; }
size_t fake_held() { return held; }
const char* fake_log() { return log_text.c_str(); }

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return status("device_sync"); }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) {
    *p = std::calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (fails("copy")) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fails("copy_async")) return cudaErrorUnknown;
    if (!sizes.count(d) || sizes[d] <= (size_t(64) << 20)) std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {  // every host buffer is pinned
    a->type = cudaMemoryTypeHost;
    a->devicePointer = const_cast<void*>(p);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    static size_t next = 1;
    *s = reinterpret_cast<cudaStream_t>(next++ % 2 + 1);  // an engine's main stream, then its side stream
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    return status(s == reinterpret_cast<cudaStream_t>(2) ? "sync main" : "sync side");
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
}

namespace pa {
bool short_geom(const BlockGeom& g) { return (g.h + 1ull) * g.out_bits <= 5ull << 31 && g.h <= 1u << 21; }
bool direct_geom(const BlockGeom& g) { return (g.h + 1ull) * g.out_bits <= 1ull << 34 && g.h <= 1u << 22; }
bool direct_overlap(const BlockGeom&, const uint32_t*, const uint32_t*) { return false; }
int make_pass_maps(const BlockGeom&, const float2*, const float2*, PassMaps*) { return 0; }
int stage_count_key_block(const BlockGeom&) { return 1; }
int kernel_count_key_block(const BlockGeom&) { return 1; }
int exact_kernel_count(const BlockGeom&) { return 1; }
int launch_publish(const void* src, void* dst, size_t bytes, cudaStream_t) {
    if (fails("publish")) return (int)cudaErrorUnknown;
    std::memcpy(dst, src, bytes);
    return 0;
}
int launch_direct(const BlockGeom&, const uint32_t*, const uint32_t*, const uint32_t*, uint32_t, uint32_t*, cudaStream_t,
                  const DirectCounts& dc) {
    if (dc.resid) *dc.resid = 0;
    return (int)status("direct");
}
int launch_seed_spectrum(const BlockGeom&, const uint32_t*, float2*, const Scratch&, unsigned long long*, int,
                         cudaStream_t) {
    return (int)status("seed");
}
int launch_key_block(const BlockGeom&, const uint32_t*, const uint32_t*, uint32_t, const float2*, const Scratch&,
                     unsigned long long*, unsigned int* resid, uint32_t*, int, cudaStream_t, cudaEvent_t*, cudaEvent_t,
                     unsigned long long*) {
    std::memcpy(resid, &residual, sizeof residual);
    return (int)status("key");
}
int launch_own_block(const BlockGeom&, const uint32_t*, const uint32_t*, const uint32_t*, uint32_t, float2*,
                     const PassMaps&, float2*, uint32_t, const Scratch&, unsigned long long*, unsigned int* resid, uint32_t*,
                     int, cudaStream_t, cudaEvent_t*, cudaEvent_t, unsigned long long*) {
    std::memcpy(resid, &residual, sizeof residual);
    return (int)status("own");
}
int launch_exact_seed(const BlockGeom&, const uint32_t*, uint32_t*, uint32_t*, cudaStream_t, unsigned long long*) {
    return (int)status("exact_seed");
}
int launch_exact_block(const BlockGeom&, const uint32_t*, const uint32_t*, const uint32_t*, uint32_t, const uint32_t*,
                       uint32_t*, uint32_t*, uint32_t*, cudaStream_t, unsigned long long*, unsigned long long*) {
    return (int)status("exact");
}
ChunkPlan chunk_plan(const BlockGeom&) { return {}; }
int chunk_kernel_count(const BlockGeom&) { return 1; }
size_t chunk_units(int log_np) { return 3 * (size_t(1) << (log_np - 27)) + 1; }
size_t chunk_staging_words(int log_np) { return ((2 * (3 + (size_t(1) << (log_np - 26))) + 2) << 21) + 64; }
void chunk_staging(int, uint32_t*, unsigned long long*, uint32_t*, ChunkBuffers*) {}
bool chunk_keeps(const ChunkPlan&, uint32_t) { return true; }
int launch_chunked_block(const BlockGeom&, const BlockGeom&, const uint32_t*, const uint32_t*, const uint32_t*, uint32_t,
                         uint32_t*, const ChunkBuffers&, bool, unsigned int*, int, cudaStream_t) {
    return (int)status("chunks");
}
}  // namespace pa

namespace pa_host {
void pool_destroy(pa_engine*) {}
}  // namespace pa_host
