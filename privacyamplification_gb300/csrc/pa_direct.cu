// pa_direct.cu -- the Toeplitz product of a short block by AND and XOR on packed words.
//
// Result bit i is XOR_j key_start[j] AND seed[(i - j) mod n]: for key word k (bits 32 k .. 32 k + 31) the seed bits
// i - 32 k - 31 .. i - 32 k are one funnel shift of two seed words, and a word step is one AND-XOR.  A lane owns
// the result bits i = lane mod 32 of M neighbouring result words, which see the same shifted seed words one key
// word later: M steps share a funnel shift.  The warps of a CTA take the key words in turn and XOR their lanes at
// the end; a lane's parity is its result bit.
//
// Up to 2^34 bit products this is faster than any transform (n = 2^18: 9.7e9 word steps of 32 bits at 64 lanes per
// clock and SM are 25 us; the transform path is some twenty launches long).
#include "pa_kernels.cuh"

namespace pa {

namespace {

constexpr int kWarps = 8;

// ONE: a single CTA takes every result word and writes them when the last is formed, for an output that
// overlaps the inputs (up to kOneWords words).
constexpr uint32_t kOneWords = 1024;
template <int M, bool ONE>
__global__ void __launch_bounds__(32 * kWarps) k_direct(const uint32_t* __restrict__ seed,
                                                        const uint32_t* __restrict__ key_start, BlockGeom g,
                                                        const uint32_t* __restrict__ key_rest, uint32_t flags,
                                                        uint32_t* __restrict__ out, uint32_t nwords) {
    __shared__ __align__(16) uint32_t sk[kWarps][32], ss[kWarps][32 + 2 * M];
    __shared__ uint32_t red[kWarps][M][32];
    __shared__ uint32_t held[ONE ? kOneWords : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (int)(g.n / 32u), kw_last = (int)(g.h / 32u);
    for (int io0 = (int)blockIdx.x * M; io0 < (int)nwords; io0 += (int)gridDim.x * M) {
        uint32_t acc[M];
#pragma unroll
        for (int m = 0; m < M; ++m) acc[m] = 0;
        for (int k0 = 32 * warp; k0 <= kw_last; k0 += 32 * kWarps) {
            // key words k0 .. k0 + 31, bit b of a word to bit b; zero past bit h (a multiple of 32)
            const int k = k0 + lane;
            uint32_t kv = 0;
            if (k < kw_last) kv = __brev(__ldg(key_start + k));
            else if (k == kw_last) kv = __ldg(key_start + k) >> 31;
            sk[warp][lane] = kv;
            // seed words io0 - k0 - 32 .. io0 - k0 + M - 1, modulo n / 32
            for (int i = lane; i < 32 + M; i += 32) {
                int q = (io0 - k0 - 32 + i) % nw;
                if (q < 0) q += nw;
                ss[warp][i] = __ldg(seed + q);
            }
            __syncwarp();
            // step u, result word m: the window of words 31 + m - u and 32 + m - u
            uint32_t w[M];  // w[m]: the window at offset m - u
#pragma unroll
            for (int m = 1; m < M; ++m) w[m - 1] = __funnelshift_lc(ss[warp][32 + m], ss[warp][31 + m], lane + 1);
#pragma unroll 8
            for (int u = 0; u < 32; ++u) {
#pragma unroll
                for (int m = M - 1; m > 0; --m) w[m] = w[m - 1];
                w[0] = __funnelshift_lc(ss[warp][32 - u], ss[warp][31 - u], lane + 1);
                const uint32_t kk = sk[warp][u];
#pragma unroll
                for (int m = 0; m < M; ++m) acc[m] ^= w[m] & kk;
            }
            __syncwarp();
        }
#pragma unroll
        for (int m = 0; m < M; ++m) red[warp][m][lane] = acc[m];
        __syncthreads();
        for (int m = warp; m < M; m += kWarps) {
            uint32_t v = 0;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) v ^= red[i][m][lane];
            const uint32_t q = (uint32_t)(io0 + m);
            const uint32_t bit = 32u * q + (uint32_t)lane;
            const uint32_t b = __ballot_sync(0xffffffffu, bit < g.out_bits && (__popc(v) & 1));
            if (lane == 0 && q < nwords) {
                uint32_t r = __brev(b);
                if ((flags & 1u) && 32u * q < g.v) r ^= __ldg(key_rest + q);
                r = __byte_perm(r, 0, 0x0123);
                if (ONE) held[q] = r;
                else out[q] = r;
            }
        }
        __syncthreads();
    }
    if (ONE)
        for (uint32_t q = threadIdx.x; q < nwords; q += 32 * kWarps) out[q] = held[q];
}

bool overlap(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + nb && y < x + na;
}

}  // namespace

bool direct_geom(const BlockGeom& g) { return ((uint64_t)g.h + 1u) * g.out_bits <= (1ull << 34); }

bool direct_overlap(const BlockGeom& g, const uint32_t* key_start, const uint32_t* out_words) {
    return overlap(out_words, 4u * (size_t)((g.out_bits + 31u) / 32u), key_start, 4u * (size_t)(g.h / 32u + 1u));
}

// Few result words: one per CTA, so that the CTAs cover the SMs; many: eight share their seed windows.  key_rest
// may be the output (a result word reads its own key_rest word only); an output over the seed or the key is
// written by one CTA at the end.
int launch_direct(const BlockGeom& g, const uint32_t* seed, const uint32_t* key_start, const uint32_t* key_rest,
                  uint32_t flags, uint32_t* out_words, cudaStream_t s) {
    const uint32_t nwords = (g.out_bits + 31u) / 32u;
    if (direct_overlap(g, key_start, out_words) || overlap(out_words, 4u * (size_t)nwords, seed, g.n / 8u)) {
        if (nwords > kOneWords) return (int)cudaErrorInvalidValue;
        k_direct<8, true><<<1, 32 * kWarps, 0, s>>>(seed, key_start, g, key_rest, flags, out_words, nwords);
    } else if (nwords <= 600u) k_direct<1, false><<<nwords, 32 * kWarps, 0, s>>>(seed, key_start, g, key_rest, flags, out_words, nwords);
    else k_direct<8, false><<<(nwords + 7u) / 8u, 32 * kWarps, 0, s>>>(seed, key_start, g, key_rest, flags, out_words, nwords);
    return (int)cudaGetLastError();
}

}  // namespace pa
