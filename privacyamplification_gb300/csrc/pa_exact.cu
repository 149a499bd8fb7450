// pa_exact.cu -- exact path: the Toeplitz product over GF(2) itself, without integers or rounding.
//
// Blocks whose FP32 residual is over the limit and calls that ask for it (PA_FLAG_EXACT) run here.  The
// result bit i is XOR_j key_start[j] AND seed[(i - j) mod n] (PrivacyAmplification.cu:740-813 rounds the
// integer convolution and takes its parity; parity is all that is kept, so it is formed directly).
//
// With K[j] = key_start[h - j] and T[m] = seed[(m - h) mod n], result bit i is XOR_j K[j] T[i + j]: the
// transpose, in the variable u, of the bilinear form sum_m T[m] (u K)[m], where u K is an ordinary product
// of polynomials over GF(2) with h + out_bits coefficients.  So with F the evaluation of a polynomial at P
// points of a field, c = F^T( (F^-T T) . (F K) ) needs transforms no longer than the product: nothing wraps,
// nothing is padded twice.
//
// Points and field.  Sequences are cut into 16-bit segments, elements of GF(2^32) through powers of z
// (pa_gf2.cuh): a product of segments has 31 coefficients and fits.  F is the additive FFT of Lin, Chung and
// Han (FOCS 2014) over a Cantor basis: conversion from monomials to products of subspace polynomials (XORs
// only, Gao and Mateer 2010), then log2 P levels of butterflies x += t y, y += x whose twiddles t, in Cantor
// coordinates, are the index bits above the butterfly's.  Level i's twiddles so lie in the subfield that
// l - 1 - i coordinates span, and the early levels multiply by GF(2), GF(4), GF(16) ... constants.  Elements
// are bit-sliced over 32 points: a product by a GF(2^16) constant costs about 8 LOP3 per element bit.
//
// What bounds it: LOP3 throughput (64 lanes per clock and SM) in the butterflies; the data of a 2^27-bit
// block is 32 MB and stays in L2.
#include "pa_gf2.cuh"
#include "pa_kernels.cuh"
#include "pa_launch.cuh"

#include <algorithm>
#include <utility>

namespace pa {

namespace {

using gf2::mul;

enum Op { kF, kT, kIT };  // transform, its transpose, the inverse of its transpose
template <Op OP>
struct OpTag {
    static constexpr Op value = OP;
};
template <int N>
struct IntTag {
    static constexpr int value = N;
};

// ============================================================================ segments <-> bit planes
// 16 words of 32 sequence bits (LSB first), two 16-bit segments each <-> 16 planes: bit e of plane p is bit p
// of segment e (e = 0 .. 31).
__device__ __forceinline__ uint32_t spread2(uint32_t x) {  // low half to the even bits, high half to the odd
    uint32_t t = (x ^ (x >> 8)) & 0x0000FF00u;
    x ^= t ^ (t << 8);
    t = (x ^ (x >> 4)) & 0x00F000F0u;
    x ^= t ^ (t << 4);
    t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
    x ^= t ^ (t << 2);
    t = (x ^ (x >> 1)) & 0x22222222u;
    return x ^ t ^ (t << 1);
}
__device__ __forceinline__ uint32_t gather2(uint32_t x) {  // the inverse
    uint32_t t = (x ^ (x >> 1)) & 0x22222222u;
    x ^= t ^ (t << 1);
    t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
    x ^= t ^ (t << 2);
    t = (x ^ (x >> 4)) & 0x00F000F0u;
    x ^= t ^ (t << 4);
    t = (x ^ (x >> 8)) & 0x0000FF00u;
    return x ^ t ^ (t << 8);
}
// Transposes the 16 x 16 bit blocks in the low and the high halves of 16 words.
__device__ __forceinline__ void transpose16(uint32_t (&w)[16]) {
    const uint32_t mask[4] = {0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int s = 8 >> k;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (!(i & s)) {
                const uint32_t t = ((w[i] >> s) ^ w[i + s]) & mask[k];
                w[i + s] ^= t;
                w[i] ^= t << s;
            }
    }
}

// Planes of the key sequence K (16 planes) or, SEED, of the windows T[16 e .. 16 e + 31] (32 planes): plane
// p's word s at V[p * pw + s] holds the elements 32 s .. 32 s + 31.
// The words of a CTA's 128 slices pass through shared memory, 17 words per slice, so that they are read in order.
constexpr int kSlices = 128;  // per CTA, one per thread
template <bool SEED>
__global__ void __launch_bounds__(kSlices) k_exact_planes(const uint32_t* __restrict__ src, BlockGeom g, uint32_t pw,
                                                          uint32_t* __restrict__ V, unsigned long long* clock) {
    __shared__ uint32_t sm[(kSlices + 1) * 17];
    pdl_wait();
    const uint32_t s = blockIdx.x * kSlices + threadIdx.x;
    if (clock && s == 0) clock_start(clock);
    const uint32_t H = g.h / 32u, nw = g.n / 32u;
    const uint64_t tbits = (uint64_t)g.h + g.out_bits;
    // word first + i of the sequence: of T, or for the key word H - q of key_start, whose top bit and the next one's
    // other bits are word q of K
    const uint64_t first = 16ull * kSlices * blockIdx.x;
    auto fetch = [&](uint32_t i) -> uint32_t {
        const uint64_t q = first + i;
        if (SEED) {
            const bool in = 32ull * q < tbits;
            const uint32_t at = q < H ? (uint32_t)q + nw - H : (uint32_t)q - H;  // (32 q - h) mod n, in words
            return in ? load(src + at) : 0u;
        }
        return q <= H ? load(src + (H - q)) : 0u;
    };
    uint32_t a[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = fetch(k * kSlices + threadIdx.x);
    uint32_t past = 0;  // the last slice's windows end in the word after the CTA's
    if (threadIdx.x == 0) past = fetch(16u * kSlices);
    auto put = [&](uint32_t i, uint32_t v) {
        if (SEED) {
            v = __brev(v);
            const uint64_t bit = 32ull * (first + i);
            if (bit < tbits && tbits - bit < 32u) v &= (1u << (tbits - bit)) - 1u;
        }
        sm[(i >> 4) * 17 + (i & 15)] = v;
    };
#pragma unroll
    for (int k = 0; k < 16; ++k) put(k * kSlices + threadIdx.x, a[k]);
    if (threadIdx.x == 0) put(16u * kSlices, past);
    __syncthreads();
    const uint32_t* w = sm + threadIdx.x * 17;  // w[17] is the next slice's first word
#pragma unroll
    for (int k = 0; k < 16; ++k)
        a[k] = SEED ? w[k] : (w[k] >> 31) | ((k < 15 ? w[k + 1] : w[17]) << 1);
    transpose16(a);
#pragma unroll
    for (int p = 0; p < 16; ++p) V[(size_t)p * pw + s] = spread2(a[p]);
    if (SEED) {
#pragma unroll
        for (int k = 0; k < 16; ++k) a[k] = __funnelshift_r(w[k], k < 15 ? w[k + 1] : w[17], 16);
        transpose16(a);
#pragma unroll
        for (int p = 0; p < 16; ++p) V[(size_t)(16 + p) * pw + s] = spread2(a[p]);
    }
}

// Planes of the result -> output words, XOR key_rest, reference byte order; written in order, as above.
__global__ void __launch_bounds__(kSlices) k_exact_words(const uint32_t* __restrict__ V, BlockGeom g, uint32_t pw,
                                                         const uint32_t* __restrict__ key_rest, uint32_t flags,
                                                         uint32_t* __restrict__ out, uint32_t nwords,
                                                         unsigned long long* clock) {
    __shared__ uint32_t sm[kSlices * 17];
    pdl_wait();
    const uint32_t s = blockIdx.x * kSlices + threadIdx.x;
    uint32_t a[16];
#pragma unroll
    for (int p = 0; p < 16; ++p) a[p] = gather2(load(V + (size_t)p * pw + s));
    transpose16(a);
#pragma unroll
    for (int k = 0; k < 16; ++k) sm[threadIdx.x * 17 + k] = a[k];
    __syncthreads();
    const uint32_t first = 16u * kSlices * blockIdx.x;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const uint32_t i = k * kSlices + threadIdx.x, q = first + i;
        if (q >= nwords) break;
        uint32_t w = sm[(i >> 4) * 17 + (i & 15)];
        const uint32_t left = g.out_bits - 32u * q;
        if (left < 32u) w &= (1u << left) - 1u;
        w = __brev(w);
        if ((flags & 1u) && 32ull * q < g.v) w ^= load(key_rest + q);
        out[q] = __byte_perm(w, 0, 0x0123);
    }
    if (clock && threadIdx.x == 0) clock_end(clock);
}

// ============================================================================ basis conversion
// One polynomial over GF(2) per plane, bit e = coefficient e.  A round (r, e) takes every run of 2^(r+1)
// coefficients as lo + x^(2^r) hi and replaces x^(2^r) by s + x^d, d = 2^e (the subspace polynomial's other
// term): hi's top d coefficients wrap into its low d, then lo += hi << d.
struct Rounds {
    int count;
    signed char r[48], e[48];
};
void add_rounds(Rounds* rs, int s, int k) {
    if (k <= 1) return;
    int t = 1;
    while (2 * t < k) t *= 2;
    for (int r = k - 1; r >= t; --r) {
        rs->r[rs->count] = (signed char)(s + r);
        rs->e[rs->count++] = (signed char)(s + r - t);
    }
    add_rounds(rs, s + t, k - t);
    add_rounds(rs, s, t);
}

// A round within a 32-bit word (R < 5).
template <int R, int E, Op OP>
__device__ __forceinline__ uint32_t word_round(uint32_t v) {
    constexpr int half = 1 << R, d = 1 << E, sh = half - d;
    constexpr uint32_t rep = R == 0 ? 0x55555555u : R == 1 ? 0x11111111u : R == 2 ? 0x01010101u : R == 3 ? 0x00010001u : 1u;
    constexpr uint32_t lowd = (1u << d) - 1u, lows = (1u << sh) - 1u;
    if (OP == kF) {
        v ^= (v >> sh) & (rep * (lowd << half));
        return v ^ ((v >> sh) & (rep * (lows << d)));
    }
    const uint32_t a = rep * (lows << half), b = rep * (lowd << (half + sh));
    if (OP == kT) {
        v ^= (v << sh) & a;
        return v ^ ((v << sh) & b);
    }
    v ^= (v << sh) & b;
    return v ^ ((v << sh) & a);
}

// Rounds on 256 coefficients held by one thread (r <= 7).
template <int R, int E, Op OP>
__device__ __forceinline__ void reg_round(uint32_t (&x)[8]) {
    if constexpr (R < 5) {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = word_round<R, E, OP>(x[i]);
    } else {
        constexpr int RW = 1 << (R - 5), DW = E >= 5 ? 1 << (E - 5) : 0, S = E >= 5 ? 0 : 1 << E;
#pragma unroll
        for (int b = 0; b < 8; b += 2 * RW) {
            uint32_t *lo = x + b, *hi = x + b + RW;
            auto wrap = [&] {
                if constexpr (OP == kF) {
                    if constexpr (DW > 0) {
#pragma unroll
                        for (int j = 0; j < DW; ++j) hi[j] ^= hi[RW - DW + j];
                    } else {
                        hi[0] ^= hi[RW - 1] >> (32 - S);
                    }
                } else if constexpr (DW > 0) {
#pragma unroll
                    for (int j = 0; j < DW; ++j) hi[RW - DW + j] ^= hi[j];
                } else {
                    hi[RW - 1] ^= hi[0] << (32 - S);
                }
            };
            auto shift = [&] {
#pragma unroll
                for (int j = 0; j < RW; ++j) {
                    if constexpr (OP == kF) {
                        if constexpr (DW > 0) {
                            if (j >= DW) lo[j] ^= hi[j - DW];
                        } else {
                            lo[j] ^= (hi[j] << S) | (j ? hi[j - 1] >> (32 - S) : 0u);
                        }
                    } else if constexpr (DW > 0) {
                        if (j + DW < RW) hi[j] ^= lo[j + DW];
                    } else {
                        hi[j] ^= (lo[j] >> S) | (j + 1 < RW ? lo[j + 1] << (32 - S) : 0u);
                    }
                }
            };
            if constexpr (OP == kT) {
                shift();
                wrap();
            } else {
                wrap();
                shift();
            }
        }
    }
}

// Rounds on 2^16 coefficients in shared memory (2048 words, NT threads), r >= 8.
constexpr int kBcThreads = 256;
template <int R, int E, Op OP>
__device__ __forceinline__ void smem_round(uint32_t* x) {
    constexpr int RW = 1 << (R - 5), DW = E >= 5 ? 1 << (E - 5) : 0, S = E >= 5 ? 0 : 1 << E;
    constexpr int NB = 1024 / RW;  // runs
    auto wrap = [&] {
        if constexpr (DW > 0) {
            for (int i = threadIdx.x; i < NB * DW; i += kBcThreads) {
                uint32_t* hi = x + (i / DW) * 2 * RW + RW;
                const int j = i % DW;
                if (OP == kF) hi[j] ^= hi[RW - DW + j];
                else hi[RW - DW + j] ^= hi[j];
            }
        } else {
            for (int i = threadIdx.x; i < NB; i += kBcThreads) {
                uint32_t* hi = x + i * 2 * RW + RW;
                if (OP == kF) hi[0] ^= hi[RW - 1] >> (32 - S);
                else hi[RW - 1] ^= hi[0] << (32 - S);
            }
        }
        __syncthreads();
    };
    auto shift = [&] {  // the loads of a thread's four pairs before the first store
        constexpr int Q = 1024 / kBcThreads;
        uint32_t v[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const int i = k * kBcThreads + (int)threadIdx.x;
            const uint32_t *lo = x + (i / RW) * 2 * RW, *hi = lo + RW;
            const int j = i % RW;
            if constexpr (OP == kF) {
                if constexpr (DW > 0) v[k] = lo[j] ^ (j >= DW ? hi[j - DW] : 0u);
                else v[k] = lo[j] ^ ((hi[j] << S) | (j ? hi[j - 1] >> (32 - S) : 0u));
            } else if constexpr (DW > 0) {
                v[k] = hi[j] ^ (j + DW < RW ? lo[j + DW] : 0u);
            } else {
                v[k] = hi[j] ^ ((lo[j] >> S) | (j + 1 < RW ? lo[j + 1] << (32 - S) : 0u));
            }
        }
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const int i = k * kBcThreads + (int)threadIdx.x;
            x[(i / RW) * 2 * RW + i % RW + (OP == kF ? 0 : RW)] = v[k];
        }
        __syncthreads();
    };
    if (OP == kT) {
        shift();
        wrap();
    } else {
        wrap();
        shift();
    }
}

// The rounds of K index bits from bit S on, in order (kT: in reverse order).
template <int K>
constexpr int split_of() {
    int t = 1;
    while (2 * t < K) t *= 2;
    return t;
}
template <int S, int K, int R, Op OP, class X>
__device__ __forceinline__ void taylor_rounds(X& x) {
    constexpr int T = split_of<K>();
    if constexpr (R >= T && R < K) {
        if constexpr (S + K <= 8) reg_round<S + R, S + R - T, OP>(x);
        else smem_round<S + R, S + R - T, OP>(x);
        taylor_rounds<S, K, OP == kT ? R + 1 : R - 1, OP>(x);
    }
}
template <int S, int K, Op OP, class X>
__device__ __forceinline__ void all_rounds(X& x) {
    if constexpr (K > 1) {
        constexpr int T = split_of<K>();
        if constexpr (OP == kT) {
            all_rounds<S, T, OP>(x);
            all_rounds<S + T, K - T, OP>(x);
            taylor_rounds<S, K, T, OP>(x);
        } else {
            taylor_rounds<S, K, K - 1, OP>(x);
            all_rounds<S + T, K - T, OP>(x);
            all_rounds<S, T, OP>(x);
        }
    }
}

// Runs of 2^16 coefficients, all their rounds: the Taylor rounds at x^256 + x and the rounds of the upper
// eight bits in shared memory, those of the lower eight bits in registers.
template <Op OP>
__global__ void __launch_bounds__(kBcThreads) k_exact_bc16(uint32_t* __restrict__ V, uint32_t pw) {
    __shared__ __align__(16) uint32_t x[2048];
    uint32_t* base = V + (size_t)blockIdx.y * pw + (size_t)blockIdx.x * 2048u;
    const int t = threadIdx.x;
    uint32_t r[8] = {};
    uint4* g4 = reinterpret_cast<uint4*>(base) + 2 * t;
    uint4* s4 = reinterpret_cast<uint4*>(x) + 2 * t;
    auto pack = [&](uint4* p) {
        p[0] = make_uint4(r[0], r[1], r[2], r[3]);
        p[1] = make_uint4(r[4], r[5], r[6], r[7]);
    };
    auto unpack = [&](const uint4* p) {
        const uint4 a = p[0], b = p[1];
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    };
    uint32_t* xp = x;
    pdl_wait();
    unpack(g4);
    if (OP == kT) all_rounds<0, 8, OP>(r);
    pack(s4);
    __syncthreads();
    if (OP == kT) {
        all_rounds<8, 8, OP>(xp);
        taylor_rounds<0, 16, 8, OP>(xp);
    } else {
        taylor_rounds<0, 16, 15, OP>(xp);
        all_rounds<8, 8, OP>(xp);
    }
    unpack(s4);
    if (OP != kT) all_rounds<0, 8, OP>(r);
    pack(g4);
}

// One round with r >= 16 over whole planes, out of place: one word per thread.
template <Op OP>
__global__ void __launch_bounds__(256) k_exact_taylor(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                      uint32_t pw, int r, int e) {
    const uint32_t w = blockIdx.x * 256u + threadIdx.x;
    if (w >= pw) return;
    pdl_wait();
    in += (size_t)blockIdx.y * pw;
    out += (size_t)blockIdx.y * pw;
    const uint32_t RW = 1u << (r - 5), o = w & (2u * RW - 1u);
    const uint32_t* lo = in + (w - o);
    const uint32_t* hi = lo + RW;
    const uint32_t DW = e >= 5 ? 1u << (e - 5) : 0u;
    const int S = e >= 5 ? 0 : 1 << e;
    uint32_t v;
    if (OP == kF) {
        auto nh = [&](uint32_t k) {  // hi after the wrap
            uint32_t x = load(hi + k);
            if (DW) {
                if (k < DW) x ^= load(hi + (RW - DW + k));
            } else if (k == 0) {
                x ^= load(hi + (RW - 1u)) >> (32 - S);
            }
            return x;
        };
        if (o >= RW) {
            v = nh(o - RW);
        } else {
            v = load(lo + o);
            if (DW) v ^= o >= DW ? nh(o - DW) : 0u;
            else v ^= (nh(o) << S) | (o ? nh(o - 1u) >> (32 - S) : 0u);
        }
    } else if (o < RW) {
        v = load(lo + o);
    } else {
        const uint32_t k = o - RW;
        auto down = [&](uint32_t j) -> uint32_t {  // lo >> d
            if (DW) return j + DW < RW ? load(lo + j + DW) : 0u;
            return (load(lo + j) >> S) | (j + 1u < RW ? load(lo + j + 1u) << (32 - S) : 0u);
        };
        auto h1 = [&](uint32_t j) { return OP == kT ? load(hi + j) ^ down(j) : load(hi + j); };
        v = h1(k);
        if (DW) {
            if (k >= RW - DW) v ^= h1(k - (RW - DW));
        } else if (k == RW - 1u) {
            v ^= h1(0) << (32 - S);
        }
        if (OP == kIT) v ^= down(k);
    }
    out[w] = v;
}

// The rounds of the index bits above 16 (the polynomial in x^65536 + x that the Taylor rounds leave): words of
// one column, R = pw / 2048 rows, in shared memory.  kBcCols columns per CTA.
constexpr uint32_t kBcCols = 16;
template <Op OP>
__global__ void __launch_bounds__(256) k_exact_bc_rows(uint32_t* __restrict__ V, uint32_t pw, Rounds rs) {
    extern __shared__ uint32_t xr[];  // [row][kBcCols]
    const uint32_t rows = pw / 2048u, c = threadIdx.x % kBcCols, r0 = threadIdx.x / kBcCols, step = 256u / kBcCols;
    uint32_t* base = V + (size_t)blockIdx.y * pw + blockIdx.x * kBcCols + c;
    pdl_wait();
    for (uint32_t i = r0; i < rows; i += step) xr[i * kBcCols + c] = base[(size_t)i * 2048u];
    __syncthreads();
    for (int k = 0; k < rs.count; ++k) {
        const int q = OP == kT ? rs.count - 1 - k : k;
        const uint32_t RW = 1u << rs.r[q], D = 1u << rs.e[q];
        auto wrap = [&] {
            for (uint32_t i = r0; i < rows / (2u * RW) * D; i += step) {
                uint32_t* hi = xr + ((i / D) * 2u * RW + RW) * kBcCols + c;
                const uint32_t j = i % D, a = j * kBcCols, b = (RW - D + j) * kBcCols;
                if (OP == kF) hi[a] ^= hi[b];
                else hi[b] ^= hi[a];
            }
            __syncthreads();
        };
        auto shift = [&] {
            for (uint32_t i = r0; i < rows / 2u; i += step) {
                uint32_t* lo = xr + (i / RW) * 2u * RW * kBcCols + c;
                uint32_t* hi = lo + RW * kBcCols;
                const uint32_t j = i % RW;
                if (OP == kF) {
                    if (j >= D) lo[j * kBcCols] ^= hi[(j - D) * kBcCols];
                } else if (j + D < RW) {
                    hi[j * kBcCols] ^= lo[(j + D) * kBcCols];
                }
            }
            __syncthreads();
        };
        if (OP == kT) {
            shift();
            wrap();
        } else {
            wrap();
            shift();
        }
    }
    for (uint32_t i = r0; i < rows; i += step) base[(size_t)i * 2048u] = xr[i * kBcCols + c];
}

// The rounds above bit 16 of up to 2^23 coefficients in one pass: R = 2^up rows of 2048 words, a tile of columns in
// shared memory.  The Taylor rounds (r, r - 16) shift a row by less than R bits in all, so that a tile needs H words
// of halo.  Leaving out the wrap, the rows grow by an overflow O_c of R - 1 bits past x^65536; reducing that once,
//   row c += x O_c + O_(c-1)
// is the same as wrapping in every round, and only the first H words of a row see it: the CTA of the first columns
// forms the overflows for itself from the last H words (kF).  Transposed, the halo is on the right, and the overflows
// O_c[k] = g_c[k + 1] + g_(c+1)[k] are what the last columns continue with (kT); undoing that (kIT) first undoes the
// rounds on the first 2 H + 1 words, which need no overflow, then runs the overflows forward and continues with those.
// The rounds among rows (the polynomial in x^65536 + x) follow or precede where `rs` has some.
// Out of place: tiles read each other's columns.  In place of one launch per Taylor round and one for the rows (52 us
// each way at 2^25 bits), and with the chain launched dependently, a 2^25-bit block takes 156 instead of 243 us.
constexpr int kUpThreads = 256;
constexpr int kMaxUp = 7;
constexpr int kUpRow = 64;   // words of a row of the tile, halo included
constexpr int kUpEdge = 16;  // words of a row of the edge tile
template <Op OP>
__global__ void __launch_bounds__(kUpThreads) k_exact_upper(const uint32_t* __restrict__ in,
                                                            uint32_t* __restrict__ out, int up, Rounds rs) {
    extern __shared__ uint32_t xu[];
    pdl_wait();
    const int R = 1 << up, H = (R + 31) / 32, W = kUpRow - H, t = threadIdx.x;
    const int w0 = (int)blockIdx.x * W, cols = min(W, 2048 - w0);  // the last tile has at least H columns
    // blockIdx.y: a run of 2^(16 + up) coefficients of some plane
    in += (size_t)blockIdx.y * (2048u << up);
    out += (size_t)blockIdx.y * (2048u << up);
    const bool edge = OP == kF ? w0 == 0 : w0 + cols == 2048;
    // tile: kF H words of halo, then the columns; otherwise the columns, then the halo.
    // edge tile: kF columns 2048 - H .. 2047 and H words past the end; otherwise columns 0 .. 2 H.
    uint32_t* xa = xu;
    uint32_t* xe = xu + R * kUpRow;
    {  // a thread's words are one column of every fourth row: four loads before the first store
        const int col = w0 + (t & (kUpRow - 1)) - (OP == kF ? H : 0);
        const bool inside = col >= 0 && col < 2048;
        for (int i0 = t; i0 < R * kUpRow; i0 += 4 * kUpThreads) {
            uint32_t v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = i0 + k * kUpThreads;
                v[k] = inside && i < R * kUpRow ? load(in + (size_t)(i / kUpRow) * 2048u + col) : 0u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i0 + k * kUpThreads < R * kUpRow) xa[i0 + k * kUpThreads] = v[k];
        }
    }
    if (edge)
        for (int i = t; i < R * kUpEdge; i += kUpThreads) {
            const int col = (i & (kUpEdge - 1)) + (OP == kF ? 2048 - H : 0);
            xe[i] = col < 2048 ? load(in + (size_t)(i / kUpEdge) * 2048u + col) : 0u;
        }
    __syncthreads();
    // Taylor rounds on words [first, last) of rows of S words: kF lo ^= hi << d, d = R/2 .. 1; otherwise
    // hi ^= lo >> d (`rising`: d from 1 up, the transpose; else from R/2 down, its inverse).  Bits from outside the
    // words count as zero.
    auto taylor = [&](uint32_t* x, auto stride, int first, int last, bool rising) {
        constexpr int S = decltype(stride)::value;
        for (int k = 0; k < up; ++k) {
            const int q = rising ? k : up - 1 - k;
            const int dw = q >= 5 ? 1 << (q - 5) : 0, bs = q >= 5 ? 0 : 1 << q;
            for (int i = t; i < (R / 2) * S; i += kUpThreads) {
                const int p = i / S, w = i & (S - 1);
                if (w < first || w >= last) continue;
                const int c = ((p >> q) << (q + 1)) | (p & ((1 << q) - 1));
                uint32_t *lo = x + c * S, *hi = lo + (S << q);
                if (OP == kF) {
                    if (bs) lo[w] ^= __funnelshift_l(w > first ? hi[w - 1] : 0u, hi[w], bs);
                    else if (w - dw >= first) lo[w] ^= hi[w - dw];
                } else {
                    if (bs) hi[w] ^= __funnelshift_r(lo[w], w + 1 < last ? lo[w + 1] : 0u, bs);
                    else if (w + dw < last) hi[w] ^= lo[w + dw];
                }
            }
            __syncthreads();
        }
    };
    // The rounds among rows, on whole rows of S words.
    auto among_rows = [&](uint32_t* x, auto stride) {
        constexpr int S = decltype(stride)::value;
        for (int k = 0; k < rs.count; ++k) {
            const int q = OP == kT ? rs.count - 1 - k : k;
            const int lr = rs.r[q], le = rs.e[q], RW = 1 << lr, D = 1 << le;
            auto wrap = [&] {
                for (int i = t; i < (R >> (lr + 1)) * D * S; i += kUpThreads) {
                    const int u = i / S, j = u & (D - 1);
                    uint32_t* hi = x + (((u >> le) << (lr + 1)) + RW) * S + (i & (S - 1));
                    if (OP == kF) hi[j * S] ^= hi[(RW - D + j) * S];
                    else hi[(RW - D + j) * S] ^= hi[j * S];
                }
                __syncthreads();
            };
            auto shift = [&] {
                for (int i = t; i < (R / 2) * S; i += kUpThreads) {
                    const int u = i / S, j = u & (RW - 1);
                    uint32_t* lo = x + ((u >> lr) << (lr + 1)) * S + (i & (S - 1));
                    uint32_t* hi = lo + RW * S;
                    if (OP == kF) {
                        if (j >= D) lo[j * S] ^= hi[(j - D) * S];
                    } else if (j + D < RW) {
                        hi[j * S] ^= lo[(j + D) * S];
                    }
                }
                __syncthreads();
            };
            if (OP == kT) {
                shift();
                wrap();
            } else {
                wrap();
                shift();
            }
        }
    };
    // Transposed overflows, from the edge tile's first words into the words after the last column.
    auto overflow = [&] {
        for (int i = t; i < R * kUpEdge; i += kUpThreads) {
            const int k = i & (kUpEdge - 1);
            if (k >= H) continue;
            const uint32_t next = i / kUpEdge + 1 < R ? xe[i + kUpEdge] : 0u;
            xa[(i / kUpEdge) * kUpRow + cols + k] = __funnelshift_r(xe[i], xe[i + 1], 1) ^ next;
        }
        __syncthreads();
    };
    using Row = IntTag<kUpRow>;
    using Edge = IntTag<kUpEdge>;
    if (OP == kF) {
        taylor(xa, Row(), 0, kUpRow, false);
        if (edge) {
            taylor(xe, Edge(), 0, 2 * H, false);
            for (int i = t; i < R * kUpEdge; i += kUpThreads) {
                const int k = i & (kUpEdge - 1);
                if (k >= H) continue;
                const uint32_t* o = xe + i + H;
                uint32_t v = (*o << 1) | (k ? o[-1] >> 31 : 0u);
                if (i >= kUpEdge) v ^= o[-kUpEdge];
                xa[(i / kUpEdge) * kUpRow + H + k] ^= v;
            }
            __syncthreads();
        }
        among_rows(xa, Row());
    } else if (OP == kT) {
        among_rows(xa, Row());
        if (edge) {
            among_rows(xe, Edge());
            overflow();
        }
        taylor(xa, Row(), 0, edge ? cols + H : kUpRow, true);
    } else {
        if (edge) {
            taylor(xe, Edge(), 0, 2 * H + 1, false);  // valid in the first H + 1 words
            overflow();
            taylor(xa, Row(), cols, cols + H, true);  // the overflows alone, through the transposed rounds
        }
        taylor(xa, Row(), 0, edge ? cols + H : kUpRow, false);
        among_rows(xa, Row());
    }
    for (int i = t; i < R * kUpRow; i += kUpThreads) {
        const int w = (i & (kUpRow - 1)) - (OP == kF ? H : 0);
        if (w >= 0 && w < cols) out[(size_t)(i / kUpRow) * 2048u + w0 + w] = xa[i];
    }
}

// ============================================================================ planes <-> field elements
// Elements: W[slice][32 words], word c = bit c of the slice's 32 elements.  A warp converts 32 slices and
// moves its 4 KB of elements through shared memory, so that both sides are coalesced.
constexpr int kRow = 36;  // words per slice in shared memory: 16-byte rows on distinct bank groups
constexpr int kConvThreads = 128;

template <bool SEED>
__global__ void __launch_bounds__(kConvThreads) k_exact_to_field(const uint32_t* __restrict__ V, uint32_t pw,
                                                                uint32_t* __restrict__ W) {
    __shared__ __align__(16) uint32_t sm[kConvThreads * kRow];
    const uint32_t s = blockIdx.x * kConvThreads + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t o[32];
    pdl_wait();
    if constexpr (SEED) {
        uint32_t in[32];
#pragma unroll
        for (int p = 0; p < 32; ++p) in[p] = load(V + (size_t)p * pw + s);
        gf2::apply<gf2::kMapTraceToField, 32, 32>(in, o);
    } else {
        uint32_t in[16];
#pragma unroll
        for (int p = 0; p < 16; ++p) in[p] = load(V + (size_t)p * pw + s);
        gf2::apply<gf2::kMapSegToField, 32, 16>(in, o);
    }
    uint4* row = reinterpret_cast<uint4*>(sm + threadIdx.x * kRow);
#pragma unroll
    for (int k = 0; k < 8; ++k) row[k] = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
    __syncwarp();
    uint4* dst = reinterpret_cast<uint4*>(W) + (size_t)(s - lane) * 8u;
    const uint32_t* wrow = sm + (threadIdx.x - lane) * kRow;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int f = 32 * k + lane;
        dst[f] = *reinterpret_cast<const uint4*>(wrow + (f >> 3) * kRow + 4 * (f & 7));
    }
}

__global__ void __launch_bounds__(kConvThreads) k_exact_to_traces(const uint32_t* __restrict__ W, uint32_t pw,
                                                                 uint32_t* __restrict__ V) {
    __shared__ __align__(16) uint32_t sm[kConvThreads * kRow];
    const uint32_t s = blockIdx.x * kConvThreads + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const uint4* src = reinterpret_cast<const uint4*>(W) + (size_t)(s - lane) * 8u;
    uint32_t* wrow = sm + (threadIdx.x - lane) * kRow;
    pdl_wait();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int f = 32 * k + lane;
        *reinterpret_cast<uint4*>(wrow + (f >> 3) * kRow + 4 * (f & 7)) = load(src + f);
    }
    __syncwarp();
    uint32_t in[32], o[16];
    const uint4* row = reinterpret_cast<const uint4*>(sm + threadIdx.x * kRow);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint4 q = row[k];
        in[4 * k] = q.x;
        in[4 * k + 1] = q.y;
        in[4 * k + 2] = q.z;
        in[4 * k + 3] = q.w;
    }
    gf2::apply<gf2::kMapFieldToTrace, 16, 32>(in, o);
#pragma unroll
    for (int p = 0; p < 16; ++p) V[(size_t)p * pw + s] = o[p];
}

// ============================================================================ butterflies
__constant__ uint32_t c_cantor[32] = {
    0x1,       0x2,       0x4,       0xa,       0x14,       0x20,       0x4c,       0xae,
    0x152,     0x22e,     0x480,     0xa4c,     0x14fa,     0x2002,     0x4c32,     0xae98,
    0x15214,   0x22e7a,   0x48066,   0xa4cc0,   0x14fa06,   0x2002ba,   0x4c3284,   0xae98d4,
    0x15294e0, 0x22eba22, 0x480d6c2, 0xa4cd0b0, 0x14fa3b2a, 0x20027c50, 0x4c325d7a, 0xae986cfa};

// Twiddle of the index bits e above a butterfly's bit (e's bit 0 is the next one up): the field element with
// Cantor coordinates 2 e, from two tables of seven bits each (e < 2^14).
struct TwiddleTables {
    uint32_t lo[128], hi[128];
    __device__ __forceinline__ uint32_t at(uint32_t e) const { return lo[e & 127u] ^ hi[e >> 7]; }
    __device__ __forceinline__ void fill() {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) {
            const int base = i < 128 ? 1 : 8;
            uint32_t v = 0;
#pragma unroll
            for (int b = 0; b < 7; ++b)
                if ((i >> b) & 1) v ^= c_cantor[base + b];
            (i < 128 ? lo : hi)[i & 127] = v;
        }
    }
};

template <int N>
__device__ __forceinline__ void load_words(const uint32_t* p, uint32_t (&v)[N]) {
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
        const uint4 q = reinterpret_cast<const uint4*>(p)[k];
        v[4 * k] = q.x;
        v[4 * k + 1] = q.y;
        v[4 * k + 2] = q.z;
        v[4 * k + 3] = q.w;
    }
}
template <int N>
__device__ __forceinline__ void store_words(uint32_t* p, const uint32_t (&v)[N]) {
#pragma unroll
    for (int k = 0; k < N / 4; ++k)
        reinterpret_cast<uint4*>(p)[k] = make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
}

// Masks of t's low K bits: b[m] all ones where bit m is set.  PRMT spreads the top bit of a byte over a word, so eight
// shifts of t serve every byte (two shifts a mask otherwise).
template <int K>
__device__ __forceinline__ void bit_masks(uint32_t t, uint32_t (&b)[K]) {
#pragma unroll
    for (int s = 0; s < 8 && s < K; ++s) {
        const int low = K < 8 ? K - 1 - s : 7 - s;  // the bit of a byte that is brought to its top
        const uint32_t v = t << (7 - low);
#pragma unroll
        for (int k = 0; 8 * k + low < K; ++k)
            asm("prmt.b32 %0, %1, 0, %2;" : "=r"(b[8 * k + low]) : "r"(v), "r"(0x8888u | 0x1111u * (uint32_t)k));
    }
}

// One butterfly on N words of x and y (shared memory) by a twiddle of GF(2^K), K <= N: its words are the masks
// of t's low K bits, XOR pat (the lane-dependent part) where PAT.
template <int K, int N, Op OP, bool PAT>
__device__ __forceinline__ void butterfly(uint32_t* px, uint32_t* py, uint32_t t, const uint32_t* pat) {
    uint32_t b[K], a[N], p[N];
    bit_masks<K>(t, b);
    if constexpr (PAT) {
        uint32_t lanes[K];
        load_words<K>(pat, lanes);
#pragma unroll
        for (int m = 0; m < K; ++m) b[m] ^= lanes[m];
    }
    load_words<N>(OP == kF ? py : px, a);
    if (OP == kT) {  // x += y first: the product's argument
        load_words<N>(py, p);
#pragma unroll
        for (int m = 0; m < N; ++m) a[m] ^= p[m];
        store_words<N>(px, a);
    }
#pragma unroll
    for (int c = 0; c < N; c += K) {
        uint32_t u[K], w[K];
#pragma unroll
        for (int m = 0; m < K; ++m) u[m] = a[c + m];
        mul<K>(u, b, w);
#pragma unroll
        for (int m = 0; m < K; ++m) p[c + m] = w[m];
    }
    uint32_t q[N];
    load_words<N>(OP == kF ? px : py, q);
#pragma unroll
    for (int m = 0; m < N; ++m) q[m] ^= p[m];
    store_words<N>(OP == kF ? px : py, q);
    if (OP != kT) {  // kF: y += x; kIT: x += y
#pragma unroll
        for (int m = 0; m < N; ++m) a[m] ^= q[m];
        store_words<N>(OP == kF ? py : px, a);
    }
}
// The same with t = 0.
template <int N, Op OP>
__device__ __forceinline__ void butterfly0(uint32_t* px, uint32_t* py) {
    uint32_t a[N], b[N];
    load_words<N>(px, a);
    load_words<N>(py, b);
#pragma unroll
    for (int m = 0; m < N; ++m) a[m] ^= b[m];
    store_words<N>(OP == kF ? py : px, a);
}

// Levels lo .. hi - 1 (T = hi - lo of them) of the transform, lo >= 5: a CTA holds the 2^T slices that differ in
// these index bits, 16 of their 32 words (every twiddle here lies in GF(2^16), so the halves are independent).
// blockIdx.x: slice below bit lo, and the half; blockIdx.y: index bits from hi up.
constexpr int kTopRow = 20;  // words per row in shared memory (16-byte rows, distinct bank groups)
template <Op OP>
__global__ void __launch_bounds__(512) k_exact_top(uint32_t* __restrict__ W, int l, int lo, int T) {
    extern __shared__ __align__(16) uint32_t xt[];
    __shared__ TwiddleTables tt;
    tt.fill();
    const uint32_t rows = 1u << T, half = blockIdx.x & 1u, col = blockIdx.x >> 1;
    const uint32_t cols = 1u << (lo - 5);
    uint32_t* base = W + ((size_t)blockIdx.y * rows * cols + col) * 32u + 16u * half;
    pdl_wait();
    {  // up to eight loads per thread (blockDim.x = rows / 2), all before the first store
        uint4 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i = k * blockDim.x + threadIdx.x;
            if (i < rows * 4u) v[k] = load(reinterpret_cast<const uint4*>(base + (size_t)(i >> 2) * cols * 32u + 4u * (i & 3u)));
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i = k * blockDim.x + threadIdx.x;
            if (i < rows * 4u) *reinterpret_cast<uint4*>(xt + (i >> 2) * kTopRow + 4u * (i & 3u)) = v[k];
        }
    }
    __syncthreads();
    for (int k = 0; k < T; ++k) {
        const int q = OP == kT ? k : T - 1 - k;  // row bit
        const int d = l - 1 - (lo + q);          // index bits above it: Cantor coordinates 1 .. d
        for (uint32_t u = threadIdx.x; u < rows / 2u; u += blockDim.x) {
            const uint32_t r = ((u >> q) << (q + 1)) | (u & ((1u << q) - 1u));
            uint32_t *px = xt + r * kTopRow, *py = px + (kTopRow << q);
            const uint32_t t = tt.at((((blockIdx.y << T) | r) >> q) >> 1);
            if (d == 0) butterfly0<16, OP>(px, py);
            else if (d == 1) butterfly<2, 16, OP, false>(px, py, t, nullptr);
            else if (d <= 3) butterfly<4, 16, OP, false>(px, py, t, nullptr);
            else if (d <= 7) butterfly<8, 16, OP, false>(px, py, t, nullptr);
            else butterfly<16, 16, OP, false>(px, py, t, nullptr);
        }
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < rows * 4u; i += blockDim.x)
        *reinterpret_cast<uint4*>(base + (size_t)(i >> 2) * cols * 32u + 4u * (i & 3u)) =
            *reinterpret_cast<const uint4*>(xt + (i >> 2) * kTopRow + 4u * (i & 3u));
}

// Levels 0 .. LOWB - 1 on 2^LOWB points.  Levels LOWB - 1 .. 5 act between slices (lanes: index bits 0 - 4);
// then every plane's 32 x 32 blocks are transposed, so that lanes are index bits 5 - 9 and the slice's low bits
// are index bits 0 - 4, and levels 4 .. 0 act between slices too, with a lane-dependent part in the twiddle.
// KEY: the key's transform, the product with the seed's (spec, in the transposed arrangement), and the
// transposed levels back.  Otherwise the seed's levels (kIT), left in the transposed arrangement.
//
// Twiddles of up to 16 coordinates lie in GF(2^16): every thread takes half of a butterfly's words.  The last
// levels of a long transform take the full product, half of the threads idle (they are other CTAs' issue slots).
template <int LOWB, bool KEY>
__global__ void __launch_bounds__(1 << (LOWB - 5), LOWB >= 13 ? 2 : 1)
    k_exact_low(uint32_t* __restrict__ W, const uint32_t* __restrict__ spec, int l) {
    constexpr int NS = 1 << (LOWB - 5), NT = NS, NB = NS / 2;
    extern __shared__ __align__(16) uint32_t xl[];  // NS rows of kRow words
    __shared__ TwiddleTables tt;
    __shared__ __align__(16) uint32_t pat[6][32];  // lane part of level i's twiddle (i < 5); zeros
    __shared__ uint32_t tc[LOWB];                  // the part of the CTA's index bits, per level
    const int t = threadIdx.x;
    uint4* g4 = reinterpret_cast<uint4*>(W) + (size_t)blockIdx.x * (NS * 8);
    tt.fill();
    for (int i = t; i < 6 * 32; i += NT) {
        const int lev = i >> 5, m = i & 31;
        uint32_t v = 0;
        if (lev < 5) {
            const uint32_t lanes[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
#pragma unroll
            for (int s = 0; s < 5; ++s)  // lane bit s is index bit 5 + s
                if ((c_cantor[5 + s - lev] >> m) & 1u) v ^= lanes[s];
        }
        pat[lev][m] = v;
    }
    if (t < LOWB) {
        uint32_t v = 0;
        for (int b = 0; b < l - LOWB; ++b)
            if ((blockIdx.x >> b) & 1u) v ^= c_cantor[LOWB + b - t];
        tc[t] = v;
    }
    pdl_wait();
    for (int f = t; f < NS * 8; f += NT) *reinterpret_cast<uint4*>(xl + (f >> 3) * kRow + 4 * (f & 7)) = g4[f];
    __syncthreads();
    // Level i between slices differing in slice bit q; transposed: after the block transposes.
    auto level = [&](auto op, int i, bool transposed) {
        constexpr Op OP = decltype(op)::value;
        const int q = transposed ? i : i - 5;
        const bool full = l - 1 - i > 15;
        const int bf = t % NB, half = t / NB;
        const uint32_t s = (uint32_t)(((bf >> q) << (q + 1)) | (bf & ((1 << q) - 1)));
        // index bits above i that the slice number gives, from bit i + 1 on
        const uint32_t e = transposed ? ((s >> 5) << (9 - i)) | ((s & 31u) >> (i + 1)) : (s >> q) >> 1;
        const uint32_t tw = tt.at(e) ^ tc[i];
        const uint32_t* pp = pat[transposed ? i : 5];  // only long transforms multiply in full before the transposes
        uint32_t* px = xl + s * kRow;
        uint32_t* py = px + (kRow << q);
        if (full) {
            if (half == 0) butterfly<32, 32, OP, true>(px, py, tw, pp);
        } else if (transposed) {
            butterfly<16, 16, OP, true>(px + 16 * half, py + 16 * half, tw, pp);
        } else {
            butterfly<16, 16, OP, false>(px + 16 * half, py + 16 * half, tw, nullptr);
        }
        __syncthreads();
    };
    // 32 x 32 bit transposes of every plane's blocks of 32 slices.
    auto transpose = [&] {
        for (int u = t; u < NS; u += NT) {
            uint32_t* b = xl + (u >> 5) * 32 * kRow + (u & 31);  // block, plane
            uint32_t w[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) w[k] = b[k * kRow];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int sh = 16 >> k;
                const uint32_t mask = k == 0   ? 0x0000FFFFu
                                      : k == 1 ? 0x00FF00FFu
                                      : k == 2 ? 0x0F0F0F0Fu
                                      : k == 3 ? 0x33333333u
                                               : 0x55555555u;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (!(j & sh)) {
                        const uint32_t x = ((w[j] >> sh) ^ w[j + sh]) & mask;
                        w[j + sh] ^= x;
                        w[j] ^= x << sh;
                    }
            }
#pragma unroll
            for (int k = 0; k < 32; ++k) b[k * kRow] = w[k];
        }
        __syncthreads();
    };
    if constexpr (KEY) {
#pragma unroll 1
        for (int i = LOWB - 1; i >= 0; --i) {
            if (i == 4) transpose();
            level(OpTag<kF>(), i, i < 5);
        }
        {  // product with the seed's transform, one slice per thread
            uint32_t a[32], b[32], c[32];
            uint32_t* px = xl + t * kRow;
            const uint4* sp = reinterpret_cast<const uint4*>(spec) + ((size_t)blockIdx.x * NS + t) * 8u;
            load_words<32>(px, a);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint4 q = load(sp + k);
                b[4 * k] = q.x;
                b[4 * k + 1] = q.y;
                b[4 * k + 2] = q.z;
                b[4 * k + 3] = q.w;
            }
            mul<32>(a, b, c);
            store_words<32>(px, c);
        }
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < LOWB; ++i) {
            level(OpTag<kT>(), i, i < 5);
            if (i == 4) transpose();
        }
    } else {
#pragma unroll 1
        for (int i = LOWB - 1; i >= 0; --i) {
            if (i == 4) transpose();
            level(OpTag<kIT>(), i, i < 5);
        }
    }
    for (int f = t; f < NS * 8; f += NT) g4[f] = *reinterpret_cast<const uint4*>(xl + (f >> 3) * kRow + 4 * (f & 7));
}

// ------------------------------------------------------------------------------------ host side
// Allows a kernel the most that any of its launches asks for.  The limit belongs to the function, not to the launch: set
// to each launch's own size, it could be lowered by another engine's thread before a longer block's launch.
template <class K>
void smem_limit(K kernel, size_t most) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}
constexpr int kMaxPoints = 27;  // log2 of the longest transform (2^30 bits, result not compressed)
constexpr int kMaxTop = 10;     // levels of one pass of k_exact_top
constexpr size_t kUpperSmem = (size_t(kUpRow + kUpEdge) << kMaxUp) * sizeof(uint32_t);
constexpr size_t kRowsSmem = (size_t(kBcCols) << (kMaxPoints - 5 - 11)) * sizeof(uint32_t);
constexpr size_t kTopSmem = (size_t(kTopRow) << kMaxTop) * sizeof(uint32_t);

// l = log2 of the points: 16 P >= h + out_bits, at least 2^16 points (the basis conversion's run).  The low
// pass takes 2^lowb points per CTA, few enough that the CTAs of a short transform cover the SMs; the levels
// above go in passes of at most 10 (80 KB of shared memory).
struct Shape {
    int l, lowb, passes, lo[2], T[2];
    uint32_t pw;  // words per plane
};
Shape shape_of(const BlockGeom& g) {
    Shape s{};
    const uint64_t need = (uint64_t)g.h + g.out_bits;
    s.l = 16;
    while ((16ull << s.l) < need) ++s.l;
    s.lowb = s.l <= 18 ? 11 : (s.l == 19 ? 12 : 13);
    const int top = s.l - s.lowb;
    s.passes = top > kMaxTop ? 2 : 1;
    s.T[0] = s.passes == 2 ? (top + 1) / 2 : top;  // the upper pass first
    s.lo[0] = s.l - s.T[0];
    s.T[1] = top - s.T[0];
    s.lo[1] = s.lowb;
    s.pw = 1u << (s.l - 5);
    return s;
}

// The launches of one transform, in order on a stream; the first error ends them.
struct Chain {
    cudaStream_t s;
    cudaError_t err = cudaSuccess;
    template <class... P, class... A>
    void run(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
        if (err == cudaSuccess) err = launch_pdl(kernel, grid, block, smem, s, std::forward<A>(args)...);
    }
};

// The basis conversion on `planes` planes in a (b: scratch of the same size); returns where the result is.
// Up to 2^23 coefficients a plane: the rounds above bit 16 in one pass; longer planes' first Taylor rounds one by one
// and the rounds among their rows in a pass of their own.
template <Op OP>
uint32_t* convert_basis(const Shape& sh, uint32_t* a, uint32_t* b, uint32_t planes, Chain& ch) {
    const int up = sh.l - 16, low = std::min(up, kMaxUp);
    Rounds rs{}, none{};
    add_rounds(&rs, 0, up);
    auto long_taylor = [&] {
        for (int k = 0; k < up - low; ++k) {
            const int r = OP == kT ? 16 + low + k : sh.l - 1 - k;
            ch.run(k_exact_taylor<OP>, dim3((sh.pw + 255u) / 256u, planes), 256, 0, a, b, sh.pw, r, r - 16);
            std::swap(a, b);
        }
    };
    auto upper = [&] {
        if (!low) return;
        const int R = 1 << low, W = kUpRow - (R + 31) / 32;
        const size_t smem = (size_t)R * (kUpRow + kUpEdge) * sizeof(uint32_t);
        smem_limit(k_exact_upper<OP>, kUpperSmem);
        ch.run(k_exact_upper<OP>, dim3((2048u + W - 1u) / W, planes << (up - low)), kUpThreads, smem, a, b, low,
               up == low ? rs : none);
        std::swap(a, b);
    };
    auto rows = [&] {
        if (up == low) return;
        const size_t smem = (size_t)(sh.pw / 2048u) * kBcCols * sizeof(uint32_t);
        smem_limit(k_exact_bc_rows<OP>, kRowsSmem);
        ch.run(k_exact_bc_rows<OP>, dim3(2048u / kBcCols, planes), 256, smem, a, sh.pw, rs);
    };
    auto runs = [&] { ch.run(k_exact_bc16<OP>, dim3(sh.pw / 2048u, planes), kBcThreads, 0, a, sh.pw); };
    if (OP == kT) {
        runs();
        rows();
        upper();
        long_taylor();
    } else {
        long_taylor();
        upper();
        rows();
        runs();
    }
    return a;
}

template <Op OP>
void top_levels(const Shape& sh, uint32_t* W, Chain& ch) {
    for (int k = 0; k < sh.passes; ++k) {
        const int p = OP == kT ? sh.passes - 1 - k : k, T = sh.T[p], lo = sh.lo[p];
        if (T == 0) continue;
        const size_t smem = ((size_t)kTopRow << T) * sizeof(uint32_t);
        smem_limit(k_exact_top<OP>, kTopSmem);
        const int nt = std::max(32, std::min(512, 1 << (T - 1)));
        ch.run(k_exact_top<OP>, dim3(2u << (lo - 5), 1u << (sh.l - lo - T)), nt, smem, W, sh.l, lo, T);
    }
}

template <int LOWB, bool KEY>
void low_levels_k(const Shape& sh, uint32_t* W, const uint32_t* spec, Chain& ch) {
    const size_t smem = ((size_t)kRow << (LOWB - 5)) * sizeof(uint32_t);
    smem_limit(k_exact_low<LOWB, KEY>, smem);
    ch.run(k_exact_low<LOWB, KEY>, 1u << (sh.l - LOWB), 1 << (LOWB - 5), smem, W, spec, sh.l);
}
template <bool KEY>
void low_levels(const Shape& sh, uint32_t* W, const uint32_t* spec, Chain& ch) {
    if (sh.lowb == 11) low_levels_k<11, KEY>(sh, W, spec, ch);
    else if (sh.lowb == 12) low_levels_k<12, KEY>(sh, W, spec, ch);
    else low_levels_k<13, KEY>(sh, W, spec, ch);
}

}  // namespace

int exact_kernel_count(const BlockGeom& g) {
    if (direct_geom(g)) return 1;
    const Shape sh = shape_of(g);
    const int up = sh.l - 16, extra = up > kMaxUp ? up - kMaxUp + 1 : 0;
    return 5 + 2 * (extra + (up ? 1 : 0) + 1 + sh.passes);
}

// Buffers: P = 2^l field elements are at most Np / 8 words, 32 planes as much.
int launch_exact_seed(const BlockGeom& g, const uint32_t* seed, uint32_t* seed_hat, uint32_t* tmp, cudaStream_t s,
                      unsigned long long* clock) {
    if (direct_geom(g)) return 0;
    const Shape sh = shape_of(g);
    Chain ch{s};
    const size_t P = size_t(32) * sh.pw;
    ch.run(k_exact_planes<true>, sh.pw / kSlices, kSlices, 0, seed, g, sh.pw, tmp, clock);
    const uint32_t* V = convert_basis<kIT>(sh, tmp, tmp + P, 32, ch);
    ch.run(k_exact_to_field<true>, sh.pw / kConvThreads, kConvThreads, 0, V, sh.pw, seed_hat);
    top_levels<kIT>(sh, seed_hat, ch);
    low_levels<false>(sh, seed_hat, nullptr, ch);
    return (int)ch.err;
}

int launch_exact_block(const BlockGeom& g, const uint32_t* seed, const uint32_t* key_start, const uint32_t* key_rest,
                       uint32_t flags, const uint32_t* seed_hat, uint32_t* a, uint32_t* tmp, uint32_t* out_words,
                       cudaStream_t s, unsigned long long* start, unsigned long long* end) {
    if (direct_geom(g)) {
        if (direct_overlap(g, key_start, out_words)) {  // every result word reads the whole key
            cudaError_t err = cudaMemcpyAsync(a, key_start, 4u * (size_t)(g.h / 32u + 1u), cudaMemcpyDeviceToDevice, s);
            if (err != cudaSuccess) return (int)err;
            key_start = a;
        }
        return launch_direct(g, seed, key_start, key_rest, flags, out_words, s, {nullptr, nullptr, 0, start});
    }
    const Shape sh = shape_of(g);
    Chain ch{s};
    const size_t half = size_t(16) * sh.pw;
    ch.run(k_exact_planes<false>, sh.pw / kSlices, kSlices, 0, key_start, g, sh.pw, tmp, start);
    const uint32_t* V = convert_basis<kF>(sh, tmp, tmp + half, 16, ch);
    ch.run(k_exact_to_field<false>, sh.pw / kConvThreads, kConvThreads, 0, V, sh.pw, a);
    top_levels<kF>(sh, a, ch);
    low_levels<true>(sh, a, seed_hat, ch);
    top_levels<kT>(sh, a, ch);
    ch.run(k_exact_to_traces, sh.pw / kConvThreads, kConvThreads, 0, a, sh.pw, tmp);
    V = convert_basis<kT>(sh, tmp, tmp + half, 16, ch);
    const uint32_t nwords = (g.out_bits + 31u) / 32u;
    ch.run(k_exact_words, ((nwords + 15u) / 16u + kSlices - 1u) / kSlices, kSlices, 0, V, g, sh.pw, key_rest, flags, out_words,
           nwords, end);
    return (int)ch.err;
}

}  // namespace pa
