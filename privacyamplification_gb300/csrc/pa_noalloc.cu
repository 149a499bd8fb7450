// pa_noalloc.cu -- pa_process_noalloc: one small block without any device allocation.
//
// Some callers cannot call cudaMalloc at all: a host whose device memory is owned by another
// allocator (a framework's caching pool that must see every byte), a latency-critical loop that may
// not take the implicit synchronisation of an allocation, or a deployment that fixes its memory map
// at start-up.  For them this entry point hashes one short block (n <= 2^15) on buffers the caller
// already owns, in one launch: the word-by-word product of pa_direct.cu, which needs no scratch and is
// exact, so that there is no residual to guard.  4096 bits: 24.4 us a call with the FP32 transforms of seed
// and key (two launches of one CTA, 9 + 17 us, and two memsets) -> 4.1 us (n = 2^15: 6.2 us).
#include "../../include/pa_gb300.h"
#include "pa_kernels.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace {

constexpr uint32_t kMaxN = 1u << 15;  // largest block (and padded cyclic length)

int ceil_log2u(uint64_t x) {
    int l = 0;
    while ((1ull << l) < x) ++l;
    return l;
}

// Geometry of a short block (same limits as the engine's single-CTA path).
int small_geom(uint32_t n, uint32_t v, uint32_t flags, pa::BlockGeom* g) {
    if (n < 1024u || (n & 31u) || (v & 31u) || v == 0 || v >= n) return PA_ERR_INVALID_ARG;
    if (n > kMaxN) return PA_ERR_TOO_LARGE;
    g->n = n;
    g->v = v;
    g->h = n - v;
    g->out_bits = (flags & PA_FLAG_COMPRESS) ? v : n / 2u;
    const bool pow2 = (n & (n - 1u)) == 0;
    if (pow2) {
        g->log_np = ceil_log2u(n);
        g->seed_direct = n;
    } else {
        g->log_np = ceil_log2u(std::max<uint64_t>(n, (uint64_t)g->out_bits + g->h));
        g->seed_direct = (uint32_t)std::min<uint64_t>((1ull << g->log_np) - g->h, n);
    }
    g->log_n = g->log_np - 1;
    g->log_n1 = g->log_n2 = 0;
    g->exact_only = 0;
    if (g->log_n > 14) return PA_ERR_TOO_LARGE;  // padded length beyond one CTA
    return PA_OK;
}

}  // namespace

extern "C" int pa_process_noalloc(const uint32_t* d_seed_words, const uint32_t* d_key_start,
                                  const uint32_t* d_key_rest, uint32_t n, uint32_t v, uint32_t flags,
                                  uint8_t* d_out, void* stream) {
    if (!d_seed_words || !d_key_start || !d_out) return PA_ERR_INVALID_ARG;
    if ((flags & PA_FLAG_XOR_KEY_REST) && !d_key_rest) return PA_ERR_INVALID_ARG;
    if (flags & PA_FLAG_EXACT) return PA_ERR_INVALID_ARG;  // a flag of the engine
    if (reinterpret_cast<uintptr_t>(d_out) & 3u) return PA_ERR_INVALID_ARG;
    pa::BlockGeom g;
    int rc = small_geom(n, v, flags, &g);
    if (rc) return rc;
    if (pa::launch_direct(g, d_seed_words, d_key_start, d_key_rest, flags, reinterpret_cast<uint32_t*>(d_out),
                          reinterpret_cast<cudaStream_t>(stream)) != 0)
        return PA_ERR_CUDA;
    return PA_OK;
}
