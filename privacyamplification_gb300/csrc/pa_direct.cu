// pa_direct.cu -- the Toeplitz product of a short block by AND and XOR on packed words.
//
// Result bit i is XOR_j key_start[j] AND seed[(i - j) mod n]: for key word k (bits 32 k .. 32 k + 31) the seed bits
// i - 32 k - 31 .. i - 32 k are one funnel shift of two seed words, and a word step is one AND-XOR.  A lane owns
// the result bits i = lane mod 32 of M neighbouring result words, which see the same shifted seed words one key
// word later: M steps share a funnel shift.  The warps of a cluster of CL CTAs take the key words in turn; their
// lanes are XORed through (distributed) shared memory at the end, and a lane's parity is its result bit.
//
// What bounds it: LOP3 and funnel shifts, 64 lanes per clock and SM (M + 1 for M word steps), and below 2^15 bits the
// launch.  On the device, kept seed, v = 3n/8, with the FP32 transforms and their two timed events -> here: 2^12 bits
// 17.0 -> 3.2 us a block, 2^14 23.1 -> 3.5, 2^15 39.5 -> 3.5, 2^16 37.0 -> 6.2, 2^17 36.8 -> 15, 1.5 2^17 31 -> 22 (2^18: 31 against
// 41, transforms).
#include "pa_kernels.cuh"
#include "pa_launch.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace pa {

namespace {

namespace cg = cooperative_groups;

constexpr int kWarps = 8;
constexpr uint32_t kOneWords = 1024;
constexpr uint32_t kCounters = 64;

// ONE: a single CTA takes every result word and writes them when the last is formed, for an output that
// overlaps the inputs (up to kOneWords words).
template <int M, int CL, bool ONE>
__global__ void __launch_bounds__(32 * kWarps, 4) k_direct(const uint32_t* __restrict__ seed,
                                                        const uint32_t* __restrict__ key_start, BlockGeom g,
                                                        const uint32_t* __restrict__ key_rest, uint32_t flags,
                                                        uint32_t* __restrict__ out, uint32_t nwords, DirectCounts dc) {
    // per warp: 32 key words, seed words 31 .. 0 of the step's 32 + M, and the M after them
    __shared__ __align__(16) uint32_t sk[kWarps][32], ss[kWarps][32], se[kWarps][M];
    __shared__ uint32_t red[kWarps][M][32];
    __shared__ uint32_t part[M][32];
    __shared__ uint32_t held[ONE ? kOneWords : 1];
    __shared__ uint32_t ones[kWarps], cta_ones;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = (int)(blockIdx.x % CL);
    const int nw = (int)(g.n / 32u), kw_last = (int)(g.h / 32u);
    const bool count = dc.cnt && blockIdx.x < CL;  // the first cluster sees every key word once
    uint32_t key_ones = 0;
    pdl_wait();
    if (dc.clock && blockIdx.x == 0 && threadIdx.x == 0) clock_start(dc.clock);
    for (int io0 = (int)(blockIdx.x / CL) * M; io0 < (int)nwords; io0 += (int)(gridDim.x / CL) * M) {
        uint32_t acc[M];
#pragma unroll
        for (int m = 0; m < M; ++m) acc[m] = 0;
        // key word k0 + lane, bit b of a word to bit b, zero past bit h (a multiple of 32); seed words
        // io0 - k0 - 32 + lane and, for lanes below M, io0 - k0 + lane, modulo n / 32 (qs and qe, stepping down)
        const int first = 32 * (rank * kWarps + warp), step = 32 * kWarps * CL, back = step % nw;
        int qs = (io0 - first - 32 + lane) % nw, qe = (io0 - first + lane) % nw;
        if (qs < 0) qs += nw;
        if (qe < 0) qe += nw;
        uint32_t kv = 0, sv = 0, ev = 0;
        auto fetch = [&](int k0) {
            const int k = k0 + lane;
            kv = 0;
            if (k < kw_last) kv = __brev(load(key_start + k));
            else if (k == kw_last) kv = load(key_start + k) >> 31;
            sv = load(seed + qs);
            if (lane < M) ev = load(seed + qe);
            qs -= back;
            qe -= back;
            if (qs < 0) qs += nw;
            if (qe < 0) qe += nw;
        };
        if (first <= kw_last) fetch(first);
        for (int k0 = first; k0 <= kw_last; k0 += step) {
            __syncwarp();
            sk[warp][lane] = kv;
            ss[warp][31 - lane] = sv;
            if (lane < M) se[warp][lane] = ev;
            key_ones += __popc(kv);
            __syncwarp();
            if (k0 + step <= kw_last) fetch(k0 + step);  // under this block's steps
            // step u, result word m: the window of seed words 31 + m - u and 32 + m - u, shifted by the lane
            uint32_t w[M], below = se[warp][0];
#pragma unroll
            for (int m = 1; m < M; ++m)
                w[m - 1] = __funnelshift_lc(se[warp][m], se[warp][m - 1], lane + 1);
#pragma unroll
            for (int u0 = 0; u0 < 32; u0 += 4) {
                const uint4 k4 = *reinterpret_cast<const uint4*>(&sk[warp][u0]);
                const uint4 s4 = *reinterpret_cast<const uint4*>(&ss[warp][u0]);
                const uint32_t kk[4] = {k4.x, k4.y, k4.z, k4.w}, sx[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
#pragma unroll
                    for (int m = M - 1; m > 0; --m) w[m] = w[m - 1];
                    w[0] = __funnelshift_lc(below, sx[u], lane + 1);
                    below = sx[u];
#pragma unroll
                    for (int m = 0; m < M; ++m) acc[m] ^= w[m] & kk[u];
                }
            }
        }
        if (count && io0 == 0) {  // this CTA's share of the key's popcount
#pragma unroll
            for (int o = 16; o; o >>= 1) key_ones += __shfl_xor_sync(0xffffffffu, key_ones, o);
            if (lane == 0) ones[warp] = key_ones;
        }
#pragma unroll
        for (int m = 0; m < M; ++m) red[warp][m][lane] = acc[m];
        __syncthreads();
        for (int m = warp; m < M; m += kWarps) {
            uint32_t v = 0;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) v ^= red[i][m][lane];
            part[m][lane] = v;
        }
        if (count && io0 == 0 && threadIdx.x == 0) {
            uint32_t t = 0;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) t += ones[i];
            cta_ones = t;
        }
        if constexpr (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
        for (int m = warp * CL + rank; m < M; m += kWarps * CL) {
            uint32_t v = 0;
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                if constexpr (CL > 1) v ^= *cg::this_cluster().map_shared_rank(&part[m][lane], c);
                else v ^= part[m][lane];
            }
            const uint32_t q = (uint32_t)(io0 + m);
            const uint32_t bit = 32u * q + (uint32_t)lane;
            const uint32_t b = __ballot_sync(0xffffffffu, bit < g.out_bits && (__popc(v) & 1));
            if (lane == 0 && q < nwords) {
                uint32_t r = __brev(b);
                if ((flags & 1u) && 32u * q < g.v) r ^= load(key_rest + q);
                r = __byte_perm(r, 0, 0x0123);
                if (ONE) held[q] = r;
                else out[q] = r;
            }
        }
        if (count && io0 == 0 && rank == 0 && threadIdx.x == 0) {
            unsigned long long t = 0;
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                if constexpr (CL > 1) t += *cg::this_cluster().map_shared_rank(&cta_ones, c);
                else t += cta_ones;
            }
            dc.cnt[0] = t;
            *dc.resid = 0u;  // nothing is rounded
        }
        if constexpr (CL > 1) cg::this_cluster().sync();  // the peers' parts are read until here
        else __syncthreads();
    }
    if (ONE)
        for (uint32_t q = threadIdx.x; q < nwords; q += 32 * kWarps) out[q] = held[q];
    // The placed seed's popcount, once per seed and placement, by up to kCounters CTAs: the last of them to add its share
    // to cnt[2] (arrivals above bit 48) takes the sum and leaves zero.  One CTA took 20 us at 2^20 bits, 270 at 2^24.
    const uint32_t counters = min(gridDim.x, kCounters);
    if (dc.count_seed && blockIdx.x < counters) {
        const uint32_t words = 1u << (g.log_np - 5);
        uint32_t c = 0;
#pragma unroll 4
        for (uint32_t w = 32 * kWarps * blockIdx.x + threadIdx.x; w < words; w += 32 * kWarps * counters)
            c += __popc(load(seed + seed_word(g, 32ull * w)));
#pragma unroll
        for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        __syncthreads();
        if (lane == 0) red[warp][0][0] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long t = 0;
            for (int i = 0; i < kWarps; ++i) t += red[i][0][0];
            const unsigned long long before = atomicAdd(dc.cnt + 2, t + (1ull << 48));
            if ((before >> 48) == counters - 1) {
                dc.cnt[1] = (before & ((1ull << 48) - 1ull)) + t;
                dc.cnt[2] = 0ull;
            }
        }
    }
    if (dc.clock && threadIdx.x == 0) clock_end(dc.clock);
}

template <int M>
struct Words {
    static constexpr int value = M;
};

bool overlap(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + nb && y < x + na;
}

}  // namespace

// The ordinary path's bounds are where the FP32 transforms (31 us from 2^17 to 2^19 bits) catch up: 9.1e9 bit products
// take 22 us, 9.7e9 26, 12.3e9 36, 16.1e9 41.  The exact path's transform takes 50 us from there on.  A long key with
// few results has few clusters and a long result with a short key few warps per CTA: the time then grows with the longer
// of the two (2^21 bits 23 .. 34 us against 34.5, 2^22 43 .. 62 against 46.5, 2^24 158 .. 172 against 98 .. 119), the
// exact path's transform being 58, 62 and 93.
static bool word_by_word(const BlockGeom& g, uint64_t products, uint64_t longest) {
    return ((uint64_t)g.h + 1u) * g.out_bits <= products && std::max(g.h, g.out_bits) <= longest;
}
bool short_geom(const BlockGeom& g) { return word_by_word(g, 5ull << 31, 1ull << 21); }
bool direct_geom(const BlockGeom& g) { return word_by_word(g, 1ull << 34, 1ull << 22); }

bool direct_overlap(const BlockGeom& g, const uint32_t* key_start, const uint32_t* out_words) {
    return overlap(out_words, 4u * (size_t)((g.out_bits + 31u) / 32u), key_start, 4u * (size_t)(g.h / 32u + 1u));
}

// Result words per cluster: four, or eight from 1200 words on (fewer funnel shifts, 2^18 bits 47.6 against 41.1 us; below,
// four keep more SMs busy).  CTAs per cluster: doubled while the CTAs number fewer than 250 and a CTA would keep 768 key
// words (2^18 bits with 163 result words: 19.4, 12.0, 9.8, 8.5 us with 1, 2, 4, 8; 2^15 bits, 96 clusters: 3.5, 4.5).
// key_rest may be the output (a result word reads its own key_rest word only); an output over the seed or the key is
// written by one CTA at the end.
int launch_direct(const BlockGeom& g, const uint32_t* seed, const uint32_t* key_start, const uint32_t* key_rest,
                  uint32_t flags, uint32_t* out_words, cudaStream_t s, const DirectCounts& dc) {
    const uint32_t nwords = (g.out_bits + 31u) / 32u, kwords = g.h / 32u + 1u;
    auto go = [&](auto kernel, uint32_t groups, uint32_t cl) {
        return (int)launch_pdl_cluster(kernel, groups * cl, 32 * kWarps, 0, s, cl, seed, key_start, g, key_rest, flags, out_words,
                               nwords, dc);
    };
    if (direct_overlap(g, key_start, out_words) || overlap(out_words, 4u * (size_t)nwords, seed, g.n / 8u)) {
        if (nwords > kOneWords) return (int)cudaErrorInvalidValue;
        return go(k_direct<8, 1, true>, 1, 1);
    }
    const uint32_t M = nwords <= 1200u ? 4u : 8u, groups = (nwords + M - 1u) / M;
    uint32_t cl = 1;
    while (cl < 8u && groups * cl < 250u && kwords >= 1536u * cl) cl *= 2u;
    auto pick = [&](auto m) {
        constexpr int W = decltype(m)::value;
        switch (cl) {
            case 1: return go(k_direct<W, 1, false>, groups, 1);
            case 2: return go(k_direct<W, 2, false>, groups, 2);
            case 4: return go(k_direct<W, 4, false>, groups, 4);
            default: return go(k_direct<W, 8, false>, groups, 8);
        }
    };
    return M == 4u ? pick(Words<4>()) : pick(Words<8>());
}

}  // namespace pa
