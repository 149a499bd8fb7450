// pa_launch.cuh -- programmatic dependent launch of a block's kernels.
//
// A block is a chain of kernels that each need the whole of the one before.  Launched with programmatic stream
// serialisation, a kernel's CTAs take the SMs as its predecessor's leave, compute their twiddle tables and set up
// their barriers, and wait in pdl_wait() for the predecessor to finish: the launch gap and the prologue run under
// the predecessor's tail.  Every kernel launched so calls pdl_wait() before its first access to data of the block,
// reads and writes alike, so that completion is transitive along the chain; in a kernel launched otherwise it does
// nothing.  The trigger is the implicit one, a CTA's exit: with an explicit one at the kernels' start, the
// successors' waiting CTAs took shared memory and warp slots from the running kernel (n = 2^27: 909 us a block
// without early launches, 922 with the explicit trigger, 897 with the implicit one; 2^20: 56.7, 48.9, 45.3 us; a
// batch of 64 uneven blocks: 6.15, 6.24, 5.94 ms).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace pa {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A block's time on the GPU's global timer: its first kernel stores the start, every CTA of its last kernel raises the
// end.  The end is not cleared (the timer only grows, so that a later block's is above it): where first and last kernel are
// one, a clear could come after another CTA's end.  Two timed events around a block took 5.5 us of the stream (2^12 bits
// 8.5 -> 3.0 us a block) and kept the next block's first kernel from being launched early.
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void clock_start(unsigned long long* clock) { clock[0] = global_ns(); }
// By one thread per CTA, after its last stores.
__device__ __forceinline__ void clock_end(unsigned long long* clock) { atomicMax(clock + 1, global_ns()); }

// Loads of the block's data in these kernels: in place of __ldg (or a plain load that the compiler may turn into one),
// whose read-only data may be fetched before the wait.
__device__ __forceinline__ uint32_t load(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float load(const float* p) { return __uint_as_float(load(reinterpret_cast<const uint32_t*>(p))); }
__device__ __forceinline__ float2 load(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 load4(const float4* p) {
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 load_stream(const float2* p) {
    float2 v;
    asm volatile("ld.global.cs.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 load(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// cluster: CTAs per cluster (x).
template <class... P, class... A>
inline cudaError_t launch_pdl_cluster(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                      unsigned cluster, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (err != cudaSuccess) cudaGetLastError();  // reported here, not by a later call
    return err;
}
template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    return launch_pdl_cluster(kernel, grid, block, smem, s, 1u, std::forward<A>(args)...);
}

}  // namespace pa
