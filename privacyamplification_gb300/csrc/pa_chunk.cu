// pa_chunk.cu -- blocks beyond the single-pass FP32 size (n > 2^27) in 2^27-bit transforms.
//
// The block's result bit i (i < out_bits) is XOR_{j <= h} key_start[j] AND T[i - j] with
// T[m] = seed[m mod n], a linear Toeplitz product.  Rows i and key positions j are cut into chunks of
// side s = 2^26; chunk (a, b) is the cyclic convolution of length n' = 2 s of key_start[b s .. b s + s) with
// T[d s, d s + s) followed by T[d s - s, d s) for d = a - b -- the technique of the reference's
// examples/LargeBlocksizeExample (GetLocalSeed / GetLocalKey / XorWithRow, main.cpp:104-124), run on the device.
// The chunks of a row are summed as spectra: every seed window and every key column is transformed forward once, a
// row's product spectrum is sum_b K_b S_(a-b), and one inverse transform per row gives the integer sums, which are
// rounded and packed straight into the result.  n = 2^29 (v = 3n/8): 7 + 5 forward and 3 inverse transforms, where
// chunk by chunk took 7 + 15 forward and 15 inverse ones: 16.7 -> 8.2 ms a block with its own seed (4.9 ms with a kept
// one, whose window spectra stay); n = 2^30 60 -> 18.5 ms.  The sums are larger than one chunk's, so the largest
// residual grows with the root of the columns: 0.021 -> 0.053 at n = 2^29, 0.074 at the most (n = 2^30, sixteen
// columns), against the limit of 0.25.
//
// Forward transforms are the row pass and the seed form of the column pass (spectra scaled by 1 / (16 Np), a power
// of two, taken back in the sum); the sum reads every spectrum once for three rows (15 x 512 MB at n = 2^29,
// bound by HBM); the inverse column pass is the second half of pass B.  Two lanes (streams with their own row-pass
// and column-pass buffers) take the transforms in turn, so that one's short kernels and tails overlap the other's.
#include "pa_pass_bodies.cuh"

#include <algorithm>

namespace pa {

namespace {

// dst = seed window d: words of T[d s, d s + s) and of T[d s - s, d s) (sw words each; indices modulo nw words).
__global__ void k_seed_window(uint32_t* __restrict__ dst, const uint32_t* __restrict__ seed, uint32_t nw, int d,
                              uint32_t sw) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 2u * sw; i += gridDim.x * blockDim.x) {
        long long src = ((long long)(i < sw ? d : d - 2) * sw + (long long)i) % (long long)nw;
        if (src < 0) src += nw;
        dst[i] = __ldg(seed + src);
    }
}

// Sum of R rows' chunk products, element by element: P_r = scale * sum_b K_b S_(a0 + r - b), b < cols.  S is a ring of
// `slots` spectra, window d in slot (d + cols) mod slots.  U: float4 (two complex values) per spectrum.
template <int R>
__global__ void __launch_bounds__(256) k_row_products(const float4* __restrict__ K, const float4* __restrict__ S,
                                                      float4* __restrict__ p0, float4* __restrict__ p1,
                                                      float4* __restrict__ p2, size_t U, int cols, int slots, int a0,
                                                      float scale) {
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * 256u + threadIdx.x;
    auto window = [&](int d) { return load4(S + (size_t)((unsigned)(d + cols) % (unsigned)slots) * U + i); };
    float4 s[R], acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r) s[r - 1] = window(a0 + r);  // shifted into place by the first step
    }
#pragma unroll 5
    for (int b = 0; b < cols; ++b) {
#pragma unroll
        for (int r = R - 1; r > 0; --r) s[r] = s[r - 1];
        s[0] = window(a0 - b);
        const float4 k = load4(K + (size_t)b * U + i);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            acc[r].x = fmaf(k.x, s[r].x, fmaf(-k.y, s[r].y, acc[r].x));
            acc[r].y = fmaf(k.x, s[r].y, fmaf(k.y, s[r].x, acc[r].y));
            acc[r].z = fmaf(k.z, s[r].z, fmaf(-k.w, s[r].w, acc[r].z));
            acc[r].w = fmaf(k.z, s[r].w, fmaf(k.w, s[r].z, acc[r].w));
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float4* p = r == 0 ? p0 : (r == 1 ? p1 : p2);
        __stcs(p + i, make_float4(acc[r].x * scale, acc[r].y * scale, acc[r].z * scale, acc[r].w * scale));
    }
}

// Popcount pairs of the rows' summed DC terms: pass C adds (cnt[0] cnt[1] / Np) mod 2, and the DC terms of a row's
// chunks add up, so cnt[0] = sum_b |K_b| |S_(a-b)| mod 2 Np, cnt[1] = 1.  Windows by slot, as above.
__global__ void k_row_counts(const unsigned long long* ck, const unsigned long long* cs, unsigned long long* row, int rows,
                             int cols, int slots, int a0, int log_np) {
    const int r = threadIdx.x;
    if (r >= rows) return;
    unsigned long long t = 0;
    for (int b = 0; b < cols; ++b) t += ck[b] * cs[(unsigned)(a0 + r - b + cols) % (unsigned)slots];
    row[2 * r] = t & ((2ull << log_np) - 1ull);
    row[2 * r + 1] = 1ull;
}

// Second half of pass B for one block of columns of 2^LOGL (two per tile): a tile's product spectrum (thread order, as
// pass B's seed form stores spectra) -> real merge, inverse column FFTs with the inverse 4-step twiddle, Z.  The
// tile's 32 values per thread come straight into registers, 512-byte runs per warp.
template <int LOGL>
__global__ void __launch_bounds__(256, 2)
    k_pass_b_inverse(const float2* __restrict__ P, float2* __restrict__ Z, BlockGeom g) {
    constexpr int L = 1 << LOGL, NT = 256, E = 32, LR = L / 16, SP = TileStride<L>::value;
    using Pl = Plan<LOGL>;
    using Lin = MapLinear<NT>;
    using TB = PassBBases<LOGL, NT>;
    constexpr int RL = Pl::RA, NSL = L / RL, QB = E / Pl::RB, QL = E / RL;
    static_assert(32 * NT / L == 2 && LR == NT && NSL == NT && QL == 2 && TB::SHARE2 && TB::SHAREL,
                  "one mirror pair of columns per tile, both of a thread's rows stored from registers");
    constexpr int U1N = 16, U2N = NSL / 16;
    extern __shared__ __align__(16) float2 sm[];  // [2][SP], then the column tables
    float2* sigma = sm + 2 * SP;                  // [2][RL]   conj(W_N^{NSL r k2})
    float2* u1 = sigma + 2 * RL;                  // [2][16]   W_N^{k2 i}
    float2* u2 = u1 + 2 * U1N;                    // [2][U2N]  W_N^{k2 16 i}
    const uint32_t n2 = 1u << g.log_n2;
    const int ntiles = (int)(n2 / 2u), t = threadIdx.x;
    float2 wb[QB], wl;
    stage_bases<L, Pl::RB, 16, +1, E, Lin>(wb);  // the same for both of the thread's butterflies
    wl = unit_root<+1>(t % NSL, NSL * RL);
    pdl_wait();
    for (int tile = (int)blockIdx.x; tile < ntiles; tile += (int)gridDim.x) {
        const float2* pt = P + (size_t)tile * (2 * L) + t;
        float2 x[E];
        // bins (k1 = t + LR r, k2 = p) and (L-1-k1, N2-p): x[r] and x[31 - r]
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            x[r] = load_stream(pt + r * LR);
            x[31 - r] = load_stream(pt + (16 + 15 - r) * LR);
        }
        __syncthreads();  // the previous tile's last reads of the exchange buffer and of the tables
        for (int i = t; i < 2 * (RL + U1N + U2N); i += NT) {
            const int c = i / (RL + U1N + U2N), j = i % (RL + U1N + U2N);
            const uint64_t k2 = col_k2((uint32_t)tile, c, n2);
            const uint64_t mult = j < RL ? (uint64_t)NSL * j : (j < RL + U1N ? (uint64_t)(j - RL) : (uint64_t)U1N * (j - RL - U1N));
            const float2 w = expmi_pi((uint32_t)(2 * ((mult * k2) & ((1ull << g.log_n) - 1))), g.log_n);
            if (j < RL) sigma[c * RL + j] = cconj(w);
            else if (j < RL + U1N) u1[c * U1N + j - RL] = w;
            else u2[c * U2N + j - RL - U1N] = w;
        }
        if (tile == 0) {  // the self-mirrored columns 0 and N2/2: pairs in natural positions, through shared memory
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                sm[padk<4>(t + LR * r)] = x[r];                      // column 0, row t + LR r
                sm[SP + padk<4>(LR - 1 - t + LR * r)] = x[16 + r];   // column 1: j = LR - 1 - t
            }
            __syncthreads();
#pragma unroll 1
            for (int u = t; u < L; u += NT) {
                int ca = 0, ka = u ? u : L / 2, kb = u ? L - u : L / 2;
                if (u >= L / 2) {
                    ca = 1;
                    ka = u - L / 2;
                    kb = L - 1 - ka;
                }
                if (u == 0) {  // Nyquist in slot (0, 0); DC is dropped
                    const float pn = sm[padk<4>(0)].x;
                    sm[padk<4>(0)] = make_float2(pn, -pn);
                }
                const float2 w = expmi_pi((uint32_t)(2 * ka + ca), LOGL + 1);  // W_2N^k, k = N2 (ka + ca / 2)
                float2 qa, qb;
                real_merge(sm[ca * SP + padk<4>(ka)], sm[ca * SP + padk<4>(kb)], w, qa, qb);
                sm[ca * SP + padk<4>(ka)] = qa;
                sm[ca * SP + padk<4>(kb)] = qb;
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                x[r] = sm[padk<4>(t + LR * r)];
                x[16 + r] = sm[SP + padk<4>(LR - 1 - t + LR * r)];
            }
        } else {
            const float2 base = expmi_pi((uint32_t)tile + n2 * (uint32_t)t, g.log_n);
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const float2 w = r ? cmul(base, make_float2(w32(r).x, -w32(r).y)) : base;
                float2 qa, qb;
                real_merge(x[r], x[31 - r], w, qa, qb);
                x[r] = qa;
                x[31 - r] = qb;
            }
        }
        stage<16, 1, +1, E>(x, nullptr);
        exchange<L, SP, 4, E, 16, 1, MapMirrorPair, Pl::RB, Lin>(x, sm);
        stage<Pl::RB, 16, +1, E>(x, wb);
        exchange<L, SP, 4, E, Pl::RB, 16, Lin, RL, Lin>(x, sm);
#pragma unroll
        for (int q = 0; q < QL; ++q) {
            const float2 c = cconj(cmul(u1[q * U1N + t % U1N], u2[q * U2N + t / U1N]));
            twiddle_powers<RL, true>(&x[q * RL], wl, c);
            dft<RL, +1>(reinterpret_cast<float2(&)[RL]>(x[q * RL]));
#pragma unroll
            for (int r = 0; r < RL; ++r) x[q * RL + r] = cmul(x[q * RL + r], sigma[q * RL + r]);
        }
        float4* Z4 = reinterpret_cast<float4*>(Z) + (size_t)tile * L;
#pragma unroll
        for (int r = 0; r < RL; ++r)
            __stcg(Z4 + t + NSL * r, make_float4(x[r].x, x[r].y, x[RL + r].x, x[RL + r].y));
    }
}

constexpr int kChunkCols = 12;  // log2 of a chunk transform's column length (rows of 2^14, the only split)

int launch_inverse(const BlockGeom& gc, const float2* P, float2* Z, int num_sms, cudaStream_t s) {
    constexpr int L = 1 << kChunkCols, RL = Plan<kChunkCols>::RA;
    constexpr size_t smem = (2 * (size_t)TileStride<L>::value + 2 * (RL + 16 + L / RL / 16)) * sizeof(float2);
    cudaFuncSetAttribute(k_pass_b_inverse<kChunkCols>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return (int)launch_pdl(k_pass_b_inverse<kChunkCols>, 2 * num_sms, 256, smem, s, P, Z, gc);
}

constexpr int kRowGroup = 3;  // rows summed in one sweep over the spectra

}  // namespace

ChunkPlan chunk_plan(const BlockGeom& g) {
    ChunkPlan p;
    p.side = 1u << kChunkLog;
    p.rows = (g.out_bits + p.side - 1u) / p.side;
    p.cols = (uint32_t)(((uint64_t)g.h + 1u + p.side - 1u) / p.side);
    // A chunk transform's key has side + 1 positions, the last one otherwise zero: when the taps past the last
    // full column are exactly one (h = cols * side, e.g. v = 3n/8), that tap takes the last column's
    // spare position instead of a column of its own.  Its seed index (i - h) lies in the column's seed
    // window like every other tap's.
    if (p.cols > 1 && ((uint64_t)g.h + 1u) % p.side == 1u) p.cols -= 1;
    p.diagonals = p.rows + p.cols - 1u;
    p.slots = std::min(p.diagonals, p.cols + (uint32_t)kRowGroup - 1u);
    return p;
}

size_t chunk_units(int log_np) { return 2 * (size_t(1) << (log_np - kChunkLog)) + kRowGroup + 2; }

size_t chunk_staging_words() {
    const size_t side = size_t(1) << kChunkLog;
    // per lane: a seed window (2 side bits); then lane 1's bit planes (Np / 8 bytes) and the popcounts
    return 2 * (2 * side / 32) + (2 * side / 32 + 64) + 256;
}

int chunk_kernel_count(const BlockGeom& g, const BlockGeom&) {
    const ChunkPlan p = chunk_plan(g);
    // window, bit rows, passes A and B per diagonal; bit rows, A, B per column; inverse, pass C, finish per row; counts
    // and products per group of rows
    return (int)(4u * p.diagonals + 3u * p.cols + 3u * p.rows + 2u * ((p.rows + kRowGroup - 1u) / kRowGroup));
}

int launch_chunked_block(const BlockGeom& g, const BlockGeom& gc, const uint32_t* seed, const uint32_t* key_start,
                         const uint32_t* key_rest, uint32_t flags, uint32_t* out_words, const ChunkBuffers& cb,
                         bool seed_ready, unsigned int* resid_bits, int num_sms, cudaStream_t s) {
    if (gc.log_n1 != kChunkCols) return (int)cudaErrorInvalidValue;
    const ChunkPlan p = chunk_plan(g);
    const uint32_t sw = p.side / 32u;
    const size_t N = size_t(1) << gc.log_n;
    const int cols = (int)p.cols, slots = (int)p.slots;
    float2* const S = cb.units;
    float2* const K = S + (size_t)slots * N;
    float2* const P2 = K + (size_t)cols * N;
    unsigned long long* const ck = cb.cnt;       // key popcounts, one per column
    unsigned long long* const cs = cb.cnt + 32;  // seed popcounts, one per slot
    unsigned long long* const crow = cb.cnt + 96;
    cudaError_t err = cudaMemsetAsync(resid_bits, 0, sizeof(unsigned int), s);
    if (err != cudaSuccess) return (int)err;
    int rc = 0;
    auto fork = [&] {
        cudaError_t e = cudaEventRecord(cb.fork, s);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(cb.lane[1].s, cb.fork, 0);
        if (!rc) rc = (int)e;
    };
    auto join = [&] {
        cudaError_t e = cudaEventRecord(cb.join, cb.lane[1].s);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s, cb.join, 0);
        if (!rc) rc = (int)e;
    };
    int turn = 0;
    auto next_lane = [&]() -> const ChunkLane& { return cb.lane[turn++ & 1]; };
    auto column_pass = [&](const ChunkLane& L, bool is_seed, unsigned long long* cnt, float2* spec) {
        if (!rc) rc = launch_pass_a(gc, L.sc.planes, is_seed, L.sc.work, cnt, num_sms, L.s);
        if (!rc) rc = launch_pass_b(gc, true, *L.sc.maps, L.sc.work, L.sc.work2, spec, L.sc.err, num_sms, L.s,
                                   kOneBlock, true);
    };
    auto seed_window = [&](int d) {
        const ChunkLane& L = next_lane();
        const int slot = (d + cols) % slots;
        k_seed_window<<<2 * num_sms, 256, 0, L.s>>>(L.window, seed, g.n / 32u, d, sw);
        if (!rc) rc = (int)cudaGetLastError();
        if (!rc) rc = launch_bit_rows(gc, L.window, true, L.sc.planes, L.s, kOneBlock, cs + slot);
        column_pass(L, true, cs + slot, S + (size_t)slot * N);
    };
    fork();
    for (int b = 0; b < cols && !rc; ++b) {
        // column b: key bits b side .. b side + side - 1, the last column up to bit h
        const ChunkLane& L = next_lane();
        BlockGeom gk = gc;
        const uint64_t first = (uint64_t)b * p.side;
        gk.h = b == cols - 1 ? (uint32_t)(g.h - first) : p.side - 1u;
        rc = launch_bit_rows(gk, key_start + first / 32u, false, L.sc.planes, L.s, kOneBlock, ck + b);
        column_pass(L, false, ck + b, K + (size_t)b * N);
    }
    if (!seed_ready)
        for (int d = -(cols - 1); d <= std::min((int)p.rows, kRowGroup) - 1 && !rc; ++d) seed_window(d);
    join();
    const float scale = (float)(16ull << gc.log_np);
    for (int a0 = 0; a0 < (int)p.rows && !rc; a0 += kRowGroup) {
        const int R = std::min(kRowGroup, (int)p.rows - a0);
        if (a0) {  // the group's new windows take the slots of the oldest
            fork();
            for (int d = a0; d < a0 + R && !rc; ++d) seed_window(d);
            join();
            if (rc) break;
        }
        // the first two rows' products in the lanes' row-pass buffers, free here
        float4* pr[3] = {reinterpret_cast<float4*>(cb.lane[0].sc.work), reinterpret_cast<float4*>(cb.lane[1].sc.work),
                         reinterpret_cast<float4*>(P2)};
        k_row_counts<<<1, 32, 0, s>>>(ck, cs, crow, R, cols, slots, a0, gc.log_np);
        const float4 *K4 = reinterpret_cast<const float4*>(K), *S4 = reinterpret_cast<const float4*>(S);
        auto products = [&](auto kernel) {
            if (!rc)
                rc = (int)launch_pdl(kernel, (unsigned)(N / 2 / 256), 256, 0, s, K4, S4, pr[0], pr[1], pr[2], N / 2, cols,
                                     slots, a0, scale);
        };
        if (R == 3) products(k_row_products<3>);
        else if (R == 2) products(k_row_products<2>);
        else products(k_row_products<1>);
        fork();
        for (int r = 0; r < R && !rc; ++r) {
            const ChunkLane& L = cb.lane[r & 1];
            const uint64_t first = (uint64_t)(a0 + r) * p.side;
            BlockGeom gr = gc;
            gr.out_bits = (uint32_t)std::min<uint64_t>(p.side, g.out_bits - first);
            gr.v = g.v > first ? (uint32_t)std::min<uint64_t>(p.side, g.v - first) : 0u;
            rc = launch_inverse(gr, reinterpret_cast<const float2*>(pr[r]), L.sc.work2, num_sms, L.s);
            if (!rc)
                rc = launch_pass_c(gr, *L.sc.maps, L.sc.work2, crow + 2 * r, L.sc.planes, resid_bits, L.sc.err, num_sms,
                                   L.s);
            if (!rc)
                rc = launch_finish(gr, L.sc.planes, key_rest ? key_rest + first / 32u : nullptr, flags,
                                   out_words + first / 32u, L.s);
        }
        join();
    }
    return rc;
}

}  // namespace pa
