// pa_engine.cu -- host side of the C ABI declared in include/pa_gb300.h.
//
// Owns the HBM working set of one GPU (the reference's device buffers di1/di2/do1/do2 and its cuFFT
// plans, PrivacyAmplification.cu:1567-1593, 1714-1751), the cached seed spectrum and the
// reuse_seed_amount bookkeeping of the host loop (PrivacyAmplification.cu:1762-1797, 2099-2101).
#include "pa_engine_impl.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

using pa::BlockGeom;
using pa_host::ceil_log2;
using pa_host::cuda_fail;
using pa_host::is_pow2;

namespace pa_host {

// Block geometry (sizes, padded cyclic length, three-pass split) for (n, v, flags).
int make_geom(uint32_t n, uint32_t v, uint32_t flags, const int8_t* split, BlockGeom* g) {
    if (n < 1024u || (n & 31u) || (v & 31u) || v == 0 || v >= n) return PA_ERR_INVALID_ARG;
    g->n = n;
    g->v = v;
    g->h = n - v;
    g->out_bits = (flags & PA_FLAG_COMPRESS) ? v : n / 2u;
    if (is_pow2(n)) {
        g->log_np = ceil_log2(n);
        g->seed_direct = n;
    } else {
        uint64_t need = std::max<uint64_t>(n, (uint64_t)g->out_bits + g->h);
        g->log_np = ceil_log2(need);
        uint64_t np = 1ull << g->log_np;
        g->seed_direct = (uint32_t)std::min<uint64_t>(np - g->h, n);
    }
    g->log_n = g->log_np - 1;
    g->exact_only = 0;
    if (g->log_n <= 14) {
        g->log_n1 = g->log_n2 = 0;
    } else if (g->log_n <= 26) {
        int l2 = split ? split[g->log_n] : 0;
        if (l2 < split_min(g->log_n) || l2 > split_max(g->log_n)) l2 = split_default(g->log_n);
        g->log_n2 = l2;  // rows 2^10..2^14, columns 2^5..2^12
        g->log_n1 = g->log_n - g->log_n2;
    } else {  // beyond the one-pass FP32 path: chunk blocks or the exact path
        g->log_n1 = g->log_n2 = 0;
        g->exact_only = 1;
        if (g->log_np > 30) return PA_ERR_TOO_LARGE;
    }
    return PA_OK;
}

bool same_seed_geom(const BlockGeom& a, const BlockGeom& b) {
    if (a.log_np != b.log_np || a.n != b.n || a.log_n2 != b.log_n2) return false;
    if (is_pow2(a.n)) return true;  // placement is the identity
    return a.seed_direct == b.seed_direct && a.h == b.h;
}

bool same_exact_geom(const BlockGeom& a, const BlockGeom& b) {
    return a.n == b.n && a.h == b.h && a.out_bits == b.out_bits;
}

}  // namespace pa_host

namespace {

using pa_host::make_geom;
using pa_host::same_exact_geom;
using pa_host::same_seed_geom;

int ensure_maps(pa_engine* e, const BlockGeom& g) {
    if (g.log_n1 == 0 || e->maps_key == pa_host::maps_key(g)) return PA_OK;
    int rc = pa::make_pass_maps(g, e->d_work, e->d_work2, &e->maps);
    if (rc) return cuda_fail(e, (cudaError_t)rc);
    e->maps_key = pa_host::maps_key(g);
    return PA_OK;
}

pa::Scratch scratch(pa_engine* e) { return {e->d_work, e->d_work2, e->d_planes, e->d_err, &e->maps}; }

int build_exact_seed(pa_engine* e, const BlockGeom& g, cudaStream_t s);

constexpr size_t kLaneUnits = 3;  // chunk buffers of lane 1: row pass, column pass, window spectrum

int build_spectrum(pa_engine* e, const BlockGeom& g, cudaStream_t s) {
    if (g.exact_only) return build_exact_seed(e, g, s);
    int rc = ensure_maps(e, g);
    if (rc) return rc;
    rc = pa::launch_seed_spectrum(g, e->d_seed, e->d_spec, scratch(e), e->d_cnt + 1, e->num_sms, s);
    if (rc) return cuda_fail(e, (cudaError_t)rc);
    e->spec_geom = g;
    e->spec_valid = true;
    return PA_OK;
}

// The seed's transform runs beside the block's: the seed serves that block only, or nothing kept can be relied on.
bool one_use(const pa_engine* e, const BlockGeom& g) {
    return (e->seed_left == 1 || e->captured) && g.log_n1 != 0 && (e->d_park || !pa::fused_geom(g));
}

// What is kept of the current seed no longer holds.
void drop_seed_data(pa_engine* e) { e->spec_valid = e->exact_valid = e->chunk_valid = e->count_valid = false; }

// A captured block may be replayed after other seeds have been set and other blocks have run.  So it transforms the seed
// that lies in d_seed then, into the buffers of the kept transforms; and since the host does not see replays, every
// block of the engine does so from then on.
int note_capture(pa_engine* e, cudaStream_t s) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    PA_CUDA(e, cudaStreamIsCapturing(s, &capture));
    if (capture != cudaStreamCaptureStatusNone) e->captured = true;
    if (e->captured) drop_seed_data(e);
    return PA_OK;
}

int seed_common(pa_engine* e, uint32_t n, int32_t reuse, cudaStream_t s) {
    e->seed_valid = true;
    e->seed_n = n;
    e->seed_left = reuse < 0 ? -1 : std::max<int64_t>(reuse, 1);
    drop_seed_data(e);
    if (is_pow2(n) && !e->captured) {  // placement does not depend on v: build the spectrum now
        BlockGeom g;
        int rc = make_geom(n, n / 2u, PA_FLAG_COMPRESS, e->split, &g);
        if (rc) return rc;
        if (g.exact_only) return PA_OK;  // chunk spectra are built per block, the exact transform on demand
        if (pa::short_geom(g)) return PA_OK;  // the block needs no spectrum, or builds it (g has the longest output)
        if (one_use(e, g)) return PA_OK;  // transformed with the block
        return build_spectrum(e, g, s);
    }
    return PA_OK;
}

// A block whose seed serves it alone (launch_own_block).  d_spec holds no spectrum that a later block could use.
int own_block(pa_engine* e, const uint32_t* d_ks, const uint32_t* d_kr, const BlockGeom& g, uint32_t flags,
                uint32_t* d_out, cudaStream_t s, cudaEvent_t* sev, cudaEvent_t kr_ready) {
    int rc = ensure_maps(e, g);
    if (rc) return rc;
    if (e->seed_maps_key != pa_host::maps_key(g)) {
        rc = pa::make_pass_maps(g, pa::fused_geom(g) ? e->d_spec : e->d_work2, e->d_work2, &e->seed_maps);
        if (rc) return cuda_fail(e, (cudaError_t)rc);
        e->seed_maps_key = pa_host::maps_key(g);
    }
    e->spec_valid = false;
    rc = pa::launch_own_block(g, e->d_seed, d_ks, d_kr, flags, e->d_spec, e->seed_maps, e->d_park, e->park_ctas,
                              scratch(e), e->d_cnt, e->d_resid, d_out, e->num_sms, s, sev, kr_ready, e->d_words->clock);
    return rc ? cuda_fail(e, (cudaError_t)rc) : PA_OK;
}

// Scratch of the exact path: 2 P words beside the P of d_work.  Engines for n > 2^27 take the second chunk lane's row-pass
// and column-pass buffers, which hold nothing from one block to the next.
uint32_t* exact_scratch(pa_engine* e) { return reinterpret_cast<uint32_t*>(e->d_chunk ? e->d_chunk : e->d_work2); }

int build_exact_seed(pa_engine* e, const BlockGeom& g, cudaStream_t s) {
    int rc = pa::launch_exact_seed(g, e->d_seed, e->d_exact_seed, exact_scratch(e), s, e->d_words->clock);
    if (rc) return cuda_fail(e, (cudaError_t)rc);
    e->exact_geom = g;
    e->exact_valid = true;
    return PA_OK;
}

// n > 2^27: the block in 2^27-bit FP32 transforms (pa_chunk.cu).  Block popcounts are not formed on this path
// (take_stats reports 0).  Lane 0 has the one-pass path's buffers and the block's stream, lane 1 the first three chunk
// buffers and `side` (free here because the block waited for key_rest's copy).  A seed that is kept has its window spectra
// kept too, where they all fit and the next block has the same rows and columns.
int chunked_block(pa_engine* e, const uint32_t* d_ks, const uint32_t* d_kr, const BlockGeom& g, uint32_t flags,
                  uint32_t* d_out, cudaStream_t s) {
    BlockGeom gc;
    const uint32_t side = 1u << pa::kChunkLog;
    int rc = make_geom(2u * side, side, 0u, e->split, &gc);
    if (rc) return rc;
    rc = ensure_maps(e, gc);
    if (rc) return rc;
    const size_t nc = size_t(1) << gc.log_n;  // complex values per buffer
    float2* const units = e->d_chunk + kLaneUnits * nc;
    if (e->lane_maps_key != pa_host::maps_key(gc)) {
        rc = pa::make_pass_maps(gc, e->d_chunk, e->d_chunk + nc, &e->lane_maps);
        for (uint32_t k = 0; k < std::min(e->chunk_count, pa::kChunkCols) && !rc; ++k)
            rc = pa::make_pass_maps(gc, units + k * nc, e->d_work2, &e->unit_maps[k]);
        if (rc) return cuda_fail(e, (cudaError_t)rc);
        e->lane_maps_key = pa_host::maps_key(gc);
    }
    pa::ChunkBuffers cb{};
    cb.lane[0].sc = scratch(e);
    cb.lane[0].spec = e->d_spec;
    cb.lane[0].s = s;
    cb.lane[1].sc = {e->d_chunk, e->d_chunk + nc, nullptr, e->d_err, &e->lane_maps};
    cb.lane[1].spec = e->d_chunk + 2 * nc;
    cb.lane[1].s = e->side;
    pa::chunk_staging(e->cap_log_np, e->d_stage, e->d_chunk_cnt, e->d_planes, &cb);
    cb.fork = e->lane_fork;
    cb.join = e->lane_join;
    cb.units = units;
    cb.count = e->chunk_count;
    cb.unit_maps = e->unit_maps;
    const pa::ChunkPlan p = pa::chunk_plan(g);
    const bool ready = e->chunk_valid && e->chunk_rows == p.rows && e->chunk_cols == p.cols;
    e->spec_valid = e->chunk_valid = false;
    rc = pa::launch_chunked_block(g, gc, e->d_seed, d_ks, d_kr, flags, d_out, cb, ready, e->d_resid, e->num_sms, s);
    if (rc) return cuda_fail(e, (cudaError_t)rc);
    e->chunk_valid = pa::chunk_keeps(p, e->chunk_count);
    e->chunk_rows = p.rows;
    e->chunk_cols = p.cols;
    return PA_OK;
}

// The stage events of one block while timing is on (null otherwise).
cudaEvent_t* stage_events(pa_engine* e, const BlockGeom& g) {
    if (!e->timing || e->tev.empty()) return nullptr;
    const size_t slot = e->tev_next;
    e->tev_stages[slot] = pa::stage_count_key_block(g);
    e->tev_next = (slot + 1) % e->tev.size();
    e->tev_count = std::min(e->tev_count + 1, e->tev.size());
    return e->tev[slot].data();
}

// A short block word by word (pa_direct.cu): exact, so that its residual is zero.  The seed's popcount is formed with
// the first block of a seed and placement.
int direct_block(pa_engine* e, const uint32_t* d_ks, const uint32_t* d_kr, const BlockGeom& g, uint32_t flags,
                 uint32_t* d_out, cudaStream_t s) {
    if (pa::direct_overlap(g, d_ks, d_out)) {  // every result word reads the whole key
        PA_CUDA(e, cudaMemcpyAsync(e->d_key_start, d_ks, (size_t)(g.h / 32u + 1u) * 4u, cudaMemcpyDeviceToDevice, s));
        d_ks = e->d_key_start;
    }
    const bool counted = e->count_valid && same_seed_geom(e->count_geom, g);
    cudaEvent_t* ev = stage_events(e, g);
    if (ev) cudaEventRecord(ev[0], s);
    int rc = pa::launch_direct(g, e->d_seed, d_ks, d_kr, flags, d_out, s,
                               {e->d_words->short_cnt, e->d_resid, counted ? 0 : 1, e->d_words->clock});
    if (rc) return cuda_fail(e, (cudaError_t)rc);
    if (ev) cudaEventRecord(ev[1], s);
    e->count_geom = g;
    e->count_valid = true;
    return PA_OK;
}

// Exact path for one block (the seed's transform is built on first use and cached with the seed).
int exact_block(pa_engine* e, const uint32_t* d_ks, const uint32_t* d_kr, const BlockGeom& g, uint32_t flags,
                uint32_t* d_out, cudaStream_t s) {
    unsigned long long* const clock = e->d_words->clock;
    unsigned long long* start = clock;  // of the seed's transform if that runs first
    if (!pa::direct_geom(g) && (!e->exact_valid || !same_exact_geom(e->exact_geom, g))) {
        int rc = build_exact_seed(e, g, s);
        if (rc) return rc;
        start = nullptr;
    }
    int rc = pa::launch_exact_block(g, e->d_seed, d_ks, d_kr, flags, e->d_exact_seed, reinterpret_cast<uint32_t*>(e->d_work),
                                    exact_scratch(e), d_out, s, start, clock);
    if (rc) return cuda_fail(e, (cudaError_t)rc);
    // the exact path leaves no residual: report 0 and the reference popcounts are not needed
    PA_CUDA(e, cudaMemsetAsync(e->d_resid, 0, sizeof(unsigned int), s));
    return PA_OK;
}

int block_common(pa_engine* e, const uint32_t* d_ks, const uint32_t* d_kr, const BlockGeom& g, uint32_t flags,
                 uint32_t* d_out, cudaStream_t s, cudaEvent_t kr_ready = nullptr) {
    if (!e->seed_valid || e->seed_left == 0) return PA_ERR_NO_SEED;
    if (g.n != e->seed_n) return PA_ERR_INVALID_ARG;
    int crc = note_capture(e, s);
    if (crc) return crc;
    e->last_chunked = e->last_direct = false;
    if (kr_ready && ((flags & PA_FLAG_EXACT) || g.exact_only))  // these paths read key_rest early
        PA_CUDA(e, cudaStreamWaitEvent(s, kr_ready, 0));
    if (flags & PA_FLAG_EXACT) {
        int rc = exact_block(e, d_ks, d_kr, g, flags, d_out, s);
        if (rc) return rc;
        e->last_exact = true;
        if (e->seed_left > 0) --e->seed_left;
        return PA_OK;
    }
    e->last_exact = false;
    if (g.exact_only) {
        PA_CUDA(e, cudaEventRecord(e->ev0, s));
        int rc = chunked_block(e, d_ks, d_kr, g, flags, d_out, s);
        if (rc) return rc;
        PA_CUDA(e, cudaEventRecord(e->ev1, s));
        e->last_chunked = true;
        if (e->seed_left > 0) --e->seed_left;
        return PA_OK;
    }
    if (pa::short_geom(g)) {
        if (kr_ready) PA_CUDA(e, cudaStreamWaitEvent(s, kr_ready, 0));
        int rc = direct_block(e, d_ks, d_kr, g, flags, d_out, s);
        if (rc) return rc;
        e->last_direct = true;
        if (e->seed_left > 0) --e->seed_left;
        return PA_OK;
    }
    const bool build = !e->spec_valid || !same_seed_geom(e->spec_geom, g), own = build && one_use(e, g);
    if (build && !own) {
        int rc = build_spectrum(e, g, s);
        if (rc) return rc;
    }
    int mrc = ensure_maps(e, g);
    if (mrc) return mrc;
    cudaEvent_t* sev = stage_events(e, g);
    if (own) {
        int rc = own_block(e, d_ks, d_kr, g, flags, d_out, s, sev, kr_ready);
        if (rc) return rc;
    } else {
        int rc = pa::launch_key_block(g, d_ks, d_kr, flags, e->d_spec, scratch(e), e->d_cnt, e->d_resid, d_out,
                                      e->num_sms, s, sev, kr_ready, e->d_words->clock);
        if (rc) return cuda_fail(e, (cudaError_t)rc);
    }
    if (e->seed_left > 0) --e->seed_left;
    return PA_OK;
}

// Statistics from the block's words on the host (h_words); `s` has finished.
int take_stats(pa_engine* e, pa_stats* st, float* resid_out) {
    const pa_engine::Words w = *e->h_words;
    if (w.err) {  // a bounded device wait expired: the block's result is not valid
        cudaMemset(e->d_err, 0, sizeof(int));
        e->last_cuda = (int)cudaErrorLaunchTimeout;
        return PA_ERR_CUDA;
    }
    float resid;
    std::memcpy(&resid, &w.resid, sizeof(resid));
    *resid_out = resid;
    if (st) {
        st->max_residual = resid;
        const bool counted = !e->last_exact && !e->last_chunked;  // short blocks and the one-pass FP32 path
        const unsigned long long* cnt = e->last_direct ? w.short_cnt : w.cnt;
        st->popcount_key = counted ? cnt[0] : 0;
        st->popcount_seed = counted ? cnt[1] : 0;
        float ms = w.clock[1] > w.clock[0] ? (float)((double)(w.clock[1] - w.clock[0]) * 1e-6) : 0.f;
        if (e->last_chunked && cudaEventElapsedTime(&ms, e->ev0, e->ev1) != cudaSuccess) {
            cudaGetLastError();  // recorded in a captured block: no time, and not an error of the next launch
            ms = 0.f;
        }
        st->gpu_ms = ms;
        st->seed_uses_left = e->seed_left < 0 ? -1 : (int32_t)e->seed_left;
        st->exact = e->last_exact ? 1 : (e->last_chunked ? 2 : 0);
    }
    return PA_OK;
}

}  // namespace

extern "C" {

size_t pa_output_bytes(uint32_t n, uint32_t v, uint32_t flags) {
    return (flags & PA_FLAG_COMPRESS) ? v / 8u : n / 16u;
}

int pa_kernels_per_block(uint32_t n, uint32_t v, uint32_t flags) {
    BlockGeom g;
    if (make_geom(n, v, flags, nullptr, &g)) return 0;
    if (flags & PA_FLAG_EXACT) return pa::exact_kernel_count(g);
    if (g.exact_only) return pa::chunk_kernel_count(g);
    return pa::kernel_count_key_block(g);
}

const char* pa_error_string(int code) {
    switch (code) {
        case PA_OK: return "ok";
        case PA_ERR_INVALID_ARG: return "invalid argument";
        case PA_ERR_CUDA: return "CUDA error";
        case PA_ERR_NO_SEED: return "no seed set or reuse_seed_amount used up";
        case PA_ERR_TOO_LARGE: return "block larger than the engine or the pool can hold";
        case PA_ERR_PRECISION: return "FP32 residual above the precision limit";
        case PA_ERR_BUSY: return "no slot or HBM free for the block now";
        case PA_PENDING: return "block still running";
        default: return "unknown error";
    }
}

int pa_last_cuda_error(pa_engine* e) { return e ? e->last_cuda : 0; }

int pa_create(const pa_config* cfg, pa_engine** out) {
    if (!cfg || !out || cfg->max_sample_size < 1024u || (cfg->max_sample_size & 31u)) return PA_ERR_INVALID_ARG;
    *out = nullptr;
    pa_engine* e = new (std::nothrow) pa_engine();
    if (!e) return PA_ERR_INVALID_ARG;
    e->device = cfg->device_id;
    e->max_n = cfg->max_sample_size;
    e->residual_limit = cfg->residual_limit > 0.f ? cfg->residual_limit : 0.25f;
    e->cap_log_np = ceil_log2(cfg->max_sample_size);
    if (e->cap_log_np > 30) {
        delete e;
        return PA_ERR_TOO_LARGE;
    }
    auto fail = [&](cudaError_t) {
        pa_destroy(e);
        return PA_ERR_CUDA;
    };
    cudaError_t err = cudaSetDevice(e->device);
    if (err != cudaSuccess) return fail(err);
    cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, e->device);
    if ((err = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking)) != cudaSuccess) return fail(err);
    if ((err = cudaEventCreate(&e->ev0)) != cudaSuccess) return fail(err);
    if ((err = cudaEventCreate(&e->ev1)) != cudaSuccess) return fail(err);
    if ((err = cudaStreamCreateWithFlags(&e->side, cudaStreamNonBlocking)) != cudaSuccess) return fail(err);
    if ((err = cudaEventCreateWithFlags(&e->kr_ready, cudaEventDisableTiming)) != cudaSuccess) return fail(err);
    if ((err = cudaEventCreateWithFlags(&e->main_ready, cudaEventDisableTiming)) != cudaSuccess) return fail(err);
    if ((err = cudaEventCreateWithFlags(&e->lane_fork, cudaEventDisableTiming)) != cudaSuccess) return fail(err);
    if ((err = cudaEventCreateWithFlags(&e->lane_join, cudaEventDisableTiming)) != cudaSuccess) return fail(err);
    size_t np = 1ull << e->cap_log_np;
    size_t words = np / 32 + 64;
    if ((err = cudaMalloc(&e->d_key_start, words * 4)) != cudaSuccess) return fail(err);
    if ((err = cudaMalloc(&e->d_key_rest, words * 4)) != cudaSuccess) return fail(err);
    if ((err = cudaMalloc(&e->d_seed, words * 4)) != cudaSuccess) return fail(err);
    if ((err = cudaMalloc(&e->d_out, words * 4)) != cudaSuccess) return fail(err);
    const size_t np_fp32 = std::min<size_t>(np, size_t(1) << 27);  // one pass of the FP32 path stops at n = 2^27
    if ((err = cudaMalloc(&e->d_work, (np_fp32 / 2) * sizeof(float2))) != cudaSuccess) return fail(err);
    if ((err = cudaMalloc(&e->d_spec, (np_fp32 / 2) * sizeof(float2))) != cudaSuccess) return fail(err);
    if ((err = cudaMalloc(&e->d_work2, (np_fp32 / 2) * sizeof(float2))) != cudaSuccess) return fail(err);
    const size_t exact_words = std::max<size_t>(np / 8, std::min<size_t>(np / 4, size_t(1) << 16));  // below 2^18: unused
    if ((err = cudaMalloc(&e->d_exact_seed, exact_words * sizeof(uint32_t))) != cudaSuccess) return fail(err);
    if ((err = cudaMalloc(&e->d_words, sizeof(pa_engine::Words))) != cudaSuccess) return fail(err);
    cudaMemset(e->d_words, 0, sizeof(pa_engine::Words));
    e->d_cnt = e->d_words->cnt;
    e->d_resid = &e->d_words->resid;
    e->d_err = &e->d_words->err;
    if ((err = cudaMallocHost((void**)&e->h_words, 64 + pa_engine::kStageBytes)) != cudaSuccess) return fail(err);
    e->h_stage = reinterpret_cast<uint8_t*>(e->h_words) + 64;
    if ((err = cudaMalloc(&e->d_planes, np_fp32 / 8 + 256)) != cudaSuccess) return fail(err);
    if (e->cap_log_np >= 21) {  // blocks with columns of 2^10 and more: the fused column pass's park
        // one spectrum tile per CTA: two CTAs per SM, at most one per tile of the largest block
        e->park_ctas = std::min<uint32_t>(2u * (uint32_t)e->num_sms, (uint32_t)((np / 2) / 8192u));
        if ((err = cudaMalloc(&e->d_park, e->park_ctas * pa::kParkBytes)) != cudaSuccess) return fail(err);
    }
    if (np > np_fp32) {
        const size_t staging = pa::chunk_staging_words(e->cap_log_np);
        if ((err = cudaMalloc(&e->d_stage, staging * sizeof(uint32_t))) != cudaSuccess) return fail(err);
        if ((err = cudaMalloc(&e->d_chunk_cnt, pa::kChunkCounts * sizeof(*e->d_chunk_cnt))) != cudaSuccess) return fail(err);
        // What is held beside lane 1's buffers only saves repeated transforms (2^29 bits: 14.0 ms a block with all of it,
        // 16.0 with none): beside other tenants of the memory it is halved until it fits.
        for (uint32_t count = (uint32_t)pa::chunk_units(e->cap_log_np);; count /= 2u) {
            e->chunk_count = count;
            err = cudaMalloc(&e->d_chunk, (kLaneUnits + count) * (np_fp32 / 2) * sizeof(float2));
            if (err == cudaSuccess) break;
            cudaGetLastError();  // reported here or not an error
            e->d_chunk = nullptr;
            if (err != cudaErrorMemoryAllocation || count == 0) return fail(err);
        }
    }
    *out = e;
    return PA_OK;
}

void pa_destroy(pa_engine* e) {
    if (!e) return;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    pa_host::pool_destroy(e);
    cudaFree(e->d_key_start);
    cudaFree(e->d_key_rest);
    cudaFree(e->d_seed);
    cudaFree(e->d_out);
    cudaFree(e->d_work);
    cudaFree(e->d_spec);
    cudaFree(e->d_exact_seed);
    cudaFree(e->d_work2);
    cudaFree(e->d_chunk);
    cudaFree(e->d_stage);
    cudaFree(e->d_chunk_cnt);
    cudaFree(e->d_words);
    cudaFreeHost(e->h_words);
    cudaFree(e->d_planes);
    cudaFree(e->d_park);
    for (auto& a : e->tev)
        for (auto ev : a) cudaEventDestroy(ev);
    if (e->ev0) cudaEventDestroy(e->ev0);
    if (e->ev1) cudaEventDestroy(e->ev1);
    if (e->kr_ready) cudaEventDestroy(e->kr_ready);
    if (e->main_ready) cudaEventDestroy(e->main_ready);
    if (e->lane_fork) cudaEventDestroy(e->lane_fork);
    if (e->lane_join) cudaEventDestroy(e->lane_join);
    if (e->side) cudaStreamDestroy(e->side);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
}

static int check_n(pa_engine* e, uint32_t n, uint32_t v, uint32_t flags, BlockGeom* g) {
    int rc = make_geom(n, v, flags, e->split, g);
    if (rc) return rc;
    if (n > e->max_n || g->log_np > e->cap_log_np) return PA_ERR_TOO_LARGE;
    return PA_OK;
}

// Seed sizes: any block size the engine accepts (the output length is only known per key block).
static int check_seed_n(pa_engine* e, uint32_t n) {
    BlockGeom g;
    return check_n(e, n, 32u, PA_FLAG_COMPRESS, &g);
}

// Waits for what a call has queued when it returns with an error: the copies and kernels read the caller's buffers.
struct WaitOnError {
    cudaStream_t main, side;
    bool ok = false;
    ~WaitOnError() {
        if (ok) return;
        cudaStreamSynchronize(side);
        cudaStreamSynchronize(main);
    }
};

int pa_set_seed(pa_engine* e, const uint32_t* seed_words, uint32_t n, int32_t reuse_seed_amount) {
    if (!e || !seed_words) return PA_ERR_INVALID_ARG;
    int rc = check_seed_n(e, n);
    if (rc) return rc;
    PA_CUDA(e, cudaSetDevice(e->device));
    WaitOnError wait{e->stream, e->side};
    PA_CUDA(e, cudaMemcpyAsync(e->d_seed, seed_words, (size_t)(n / 32u) * 4u, cudaMemcpyHostToDevice, e->stream));
    rc = seed_common(e, n, reuse_seed_amount, e->stream);
    if (rc) return rc;
    PA_CUDA(e, cudaStreamSynchronize(e->stream));
    wait.ok = true;
    return PA_OK;
}

int pa_set_seed_device(pa_engine* e, const uint32_t* d_seed_words, uint32_t n, int32_t reuse_seed_amount,
                       void* stream) {
    if (!e || !d_seed_words) return PA_ERR_INVALID_ARG;
    int rc = check_seed_n(e, n);
    if (rc) return rc;
    cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
    PA_CUDA(e, cudaSetDevice(e->device));
    rc = note_capture(e, s);
    if (rc) return rc;
    PA_CUDA(e, cudaMemcpyAsync(e->d_seed, d_seed_words, (size_t)(n / 32u) * 4u, cudaMemcpyDeviceToDevice, s));
    e->pending = true;
    return seed_common(e, n, reuse_seed_amount, s);
}

// Device address of pinned (or registered) host memory that kernels can read in 32-bit words, else null.
static const uint32_t* pinned_view(const uint32_t* p) {
    cudaPointerAttributes at{};
    if ((reinterpret_cast<uintptr_t>(p) & 3u) || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return at.type == cudaMemoryTypeHost ? static_cast<const uint32_t*>(at.devicePointer) : nullptr;
}

int pa_process(pa_engine* e, const uint32_t* key_start, const uint32_t* key_rest, uint32_t n, uint32_t v,
               uint32_t flags, uint8_t* out, pa_stats* stats) {
    if (!e || !key_start || !out) return PA_ERR_INVALID_ARG;
    if ((flags & PA_FLAG_XOR_KEY_REST) && !key_rest) return PA_ERR_INVALID_ARG;
    BlockGeom g;
    int rc = check_n(e, n, v, flags, &g);
    if (rc) return rc;
    if (!e->seed_valid || e->seed_left == 0) return PA_ERR_NO_SEED;
    if (n != e->seed_n) return PA_ERR_INVALID_ARG;
    PA_CUDA(e, cudaSetDevice(e->device));
    cudaStream_t s = e->stream;
    WaitOnError wait{s, e->side};
    // Pinned inputs of up to 256 KB are read where they lie: a copy of any size holds the stream for 11 us (2^16 bits
    // host to host 40 -> 29.5 us a call; longer keys come faster by a copy).  A transform reads the key once (2^18 .. 2^22
    // bits, keys of 3 to 230 KB: 1 to 4 us a call less than with a copy); a word-by-word block reads it once per cluster
    // of CTAs, mostly from cache, which is level with a copy or faster up to 32 KB and slower from 64 KB on (128 KB 41 us
    // against 36, 256 KB 58 against 48).  key_rest is first read by the block's last kernel: a long one is copied on the side stream
    // (after whatever the engine stream had queued) while the passes run.
    const bool reread = (flags & PA_FLAG_EXACT) ? pa::direct_geom(g) : pa::short_geom(g);
    const size_t ks_bytes = (size_t)(g.h / 32u + 1u) * 4u;
    const uint32_t* d_ks = ks_bytes <= (reread ? pa_engine::kRereadBytes : pa_engine::kStageBytes) ? pinned_view(key_start)
                                                                                                   : nullptr;
    if (!d_ks) {
        PA_CUDA(e, cudaMemcpyAsync(e->d_key_start, key_start, ks_bytes, cudaMemcpyHostToDevice, s));
        d_ks = e->d_key_start;
    }
    cudaEvent_t kr_ready = nullptr;
    const uint32_t* d_kr = e->d_key_rest;
    const size_t kr_bytes = (size_t)(v / 32u) * 4u;
    if ((flags & PA_FLAG_XOR_KEY_REST) && kr_bytes <= pa_engine::kStageBytes) {
        d_kr = pinned_view(key_rest);
        if (!d_kr) {
            PA_CUDA(e, cudaMemcpyAsync(e->d_key_rest, key_rest, kr_bytes, cudaMemcpyHostToDevice, s));
            d_kr = e->d_key_rest;
        }
    } else if (flags & PA_FLAG_XOR_KEY_REST) {
        PA_CUDA(e, cudaEventRecord(e->main_ready, s));
        PA_CUDA(e, cudaStreamWaitEvent(e->side, e->main_ready, 0));
        PA_CUDA(e, cudaMemcpyAsync(e->d_key_rest, key_rest, kr_bytes, cudaMemcpyHostToDevice, e->side));
        PA_CUDA(e, cudaEventRecord(e->kr_ready, e->side));
        kr_ready = e->kr_ready;
    }
    // A short result goes to pinned staging, and the block's words follow it by a kernel; both are waited for once, and
    // the caller's buffer is written when the words say that the result holds.
    const size_t ob = pa_output_bytes(n, v, flags);
    const bool staged = ob <= pa_engine::kStageBytes;
    uint32_t* const d_out = staged ? reinterpret_cast<uint32_t*>(e->h_stage) : e->d_out;
    rc = block_common(e, d_ks, d_kr, g, flags, d_out, s, kr_ready);
    if (rc) return rc;
    auto collect = [&](pa_stats* st, float* resid) -> int {
        int prc = pa::launch_publish(e->d_words, e->h_words, sizeof(pa_engine::Words), s);
        if (prc) return cuda_fail(e, (cudaError_t)prc);
        PA_CUDA(e, cudaStreamSynchronize(s));
        return take_stats(e, st, resid);
    };
    float resid = 0.f;
    rc = collect(stats, &resid);
    if (rc) return rc;
    if (!(resid <= e->residual_limit)) {
        // FP32 rounding budget exceeded: recompute this block exactly (same inputs, same seed use)
        if (e->seed_left >= 0) ++e->seed_left;
        rc = block_common(e, d_ks, d_kr, g, flags | PA_FLAG_EXACT, d_out, s);
        if (rc) return rc;
        float r2 = 0.f;
        rc = collect(stats, &r2);
        if (rc) return rc;
        if (stats) stats->max_residual = resid;  // report what the FP32 path measured
    }
    if (staged) std::memcpy(out, e->h_stage, ob);
    else PA_CUDA(e, cudaMemcpy(out, e->d_out, ob, cudaMemcpyDeviceToHost));
    wait.ok = true;
    return PA_OK;
}

int pa_process_device(pa_engine* e, const uint32_t* d_key_start, const uint32_t* d_key_rest, uint32_t n, uint32_t v,
                      uint32_t flags, uint8_t* d_out, void* stream) {
    if (!e || !d_key_start || !d_out) return PA_ERR_INVALID_ARG;
    if ((flags & PA_FLAG_XOR_KEY_REST) && !d_key_rest) return PA_ERR_INVALID_ARG;
    if (reinterpret_cast<uintptr_t>(d_out) & 3u) return PA_ERR_INVALID_ARG;
    BlockGeom g;
    int rc = check_n(e, n, v, flags, &g);
    if (rc) return rc;
    cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
    PA_CUDA(e, cudaSetDevice(e->device));
    e->pending = true;
    return block_common(e, d_key_start, d_key_rest, g, flags, reinterpret_cast<uint32_t*>(d_out), s);
}

int pa_sync(pa_engine* e, pa_stats* stats) {
    if (!e) return PA_ERR_INVALID_ARG;
    PA_CUDA(e, cudaSetDevice(e->device));
    PA_CUDA(e, cudaDeviceSynchronize());
    e->pending = false;
    PA_CUDA(e, cudaMemcpy(e->h_words, e->d_words, sizeof(pa_engine::Words), cudaMemcpyDeviceToHost));
    float resid = 0.f;
    int rc = take_stats(e, stats, &resid);
    if (rc) return rc;
    return resid <= e->residual_limit ? PA_OK : PA_ERR_PRECISION;
}

int pa_set_timing(pa_engine* e, int enable) {
    if (!e) return PA_ERR_INVALID_ARG;
    PA_CUDA(e, cudaSetDevice(e->device));
    if (enable && e->tev.empty()) {
        const size_t slots = 1024;
        e->tev.resize(slots);
        e->tev_stages.assign(slots, 0);
        for (auto& a : e->tev)
            for (auto& ev : a) PA_CUDA(e, cudaEventCreate(&ev));
    }
    e->timing = enable != 0;
    e->tev_next = e->tev_count = 0;
    return PA_OK;
}

int pa_stage_times(pa_engine* e, float* ms, int max_stages, int* nstages, int* nblocks) {
    if (!e || !ms || max_stages <= 0) return PA_ERR_INVALID_ARG;
    PA_CUDA(e, cudaSetDevice(e->device));
    double acc[4] = {0, 0, 0, 0};
    int stages = 0, blocks = 0;
    size_t n = e->tev_count, first = (e->tev_next + e->tev.size() - n) % std::max<size_t>(1, e->tev.size());
    for (size_t k = 0; k < n; ++k) {
        size_t slot = (first + k) % e->tev.size();
        int st = e->tev_stages[slot];
        if (blocks && st != stages) continue;  // average blocks of one shape only
        stages = st;
        PA_CUDA(e, cudaEventSynchronize(e->tev[slot][st]));
        for (int i = 0; i < st; ++i) {
            float t = 0.f;
            PA_CUDA(e, cudaEventElapsedTime(&t, e->tev[slot][i], e->tev[slot][i + 1]));
            acc[i] += t;
        }
        ++blocks;
    }
    for (int i = 0; i < std::min(stages, max_stages); ++i) ms[i] = blocks ? (float)(acc[i] / blocks) : 0.f;
    if (nstages) *nstages = stages;
    if (nblocks) *nblocks = blocks;
    e->tev_next = e->tev_count = 0;
    return PA_OK;
}

int pa_key_split(const uint32_t* recv_key, uint32_t n, uint32_t v, uint32_t* key_start, uint32_t* key_rest) {
    if (!recv_key || !key_start || !key_rest || (n & 31u) || (v & 31u) || v == 0 || v >= n)
        return PA_ERR_INVALID_ARG;
    uint32_t hb = (n - v) / 32u, vb = v / 32u, nb = n / 32u;
    std::memset(key_start, 0, (size_t)nb * 4u);
    std::memcpy(key_start, recv_key, (size_t)hb * 4u);
    key_start[hb] = recv_key[hb] & 0x80000000u;
    for (uint32_t i = 0; i < vb; ++i) key_rest[i] = (recv_key[hb + i] << 1) | (recv_key[hb + i + 1] >> 31);
    return PA_OK;
}

}  // extern "C"
