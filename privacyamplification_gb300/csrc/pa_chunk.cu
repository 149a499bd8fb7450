// pa_chunk.cu -- blocks beyond the single-pass FP32 size (n > 2^27) in 2^27-bit transforms.
//
// The block's result bit i (i < out_bits) is XOR_{j <= h} key_start[j] AND T[i - j] with
// T[m] = seed[m mod n], a linear Toeplitz product.  Rows i and key positions j are cut into chunks of
// side s = 2^26; chunk (a, b) is the cyclic convolution of length n' = 2 s of key_start[b s .. b s + s) with
// T[d s, d s + s) followed by T[d s - s, d s) for d = a - b -- the technique of the reference's
// examples/LargeBlocksizeExample (GetLocalSeed / GetLocalKey / XorWithRow, main.cpp:104-124), run on the device.
// The chunks of a diagonal d share a seed window and its spectrum, those of a column the key's row pass, which is
// kept for the block: n = 2^29 (v = 3n/8) takes 7 seed transforms, 5 row passes of the key and 15 column and inverse row
// passes, 14.0 ms a block (10.5 with a kept seed, whose window spectra stay; 16.7 with the key's row pass in every chunk).
// Every chunk is rounded by itself and the rows are XORed, so that the FP32 error is one chunk's: largest residual 0.022 at
// n = 2^29, 0.021 for a single chunk.  Summing a row's chunks as spectra and rounding once takes 3 inverse transforms in
// place of 15, 8.2 ms, but the error grows with the root of the columns (0.053, and 0.074 at 2^30), and structured blocks
// that are within the limit chunk by chunk are not within it as a sum.
//
// Two lanes (streams with their own buffers) take the diagonals in turn, so that one's short kernels and tails overlap
// the other's.
#include "pa_kernels.cuh"
#include "pa_launch.cuh"

#include <algorithm>

namespace pa {

namespace {

constexpr uint32_t kXorFlag = 1u;  // PA_FLAG_XOR_KEY_REST
constexpr uint32_t kSide = 1u << kChunkLog, kSideWords = kSide / 32u;

// dst = seed window d: words of T[d s, d s + s) and of T[d s - s, d s) (indices modulo nw words).
__global__ void k_seed_window(uint32_t* __restrict__ dst, const uint32_t* __restrict__ seed, uint32_t nw, int d) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 2u * kSideWords; i += gridDim.x * blockDim.x) {
        long long src = ((long long)(i < kSideWords ? d : d - 2) * kSideWords + (long long)i) % (long long)nw;
        if (src < 0) src += nw;
        dst[i] = __ldg(seed + src);
    }
}

// Popcount pairs (key column, seed window) as pass C reads them; columns from `held` on get their key's later.
__global__ void k_chunk_counts(unsigned long long* pairs, const unsigned long long* key, const unsigned long long* window,
                               int held) {
    const int b = threadIdx.x;
    if (b < held) pairs[2 * b] = key[b];
    pairs[2 * b + 1] = *window;
}

__global__ void k_xor_rows(uint4* __restrict__ acc, const uint4* __restrict__ add, uint32_t quads) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += gridDim.x * blockDim.x) {
        const uint4 x = acc[i], y = add[i];
        acc[i] = make_uint4(x.x ^ y.x, x.y ^ y.y, x.z ^ y.z, x.w ^ y.w);
    }
}

// Output words = the lanes' rows XOR key_rest (byte-swapped words).  A lane has row a if bit a of its mask is set.
__global__ void k_chunk_final(uint32_t* __restrict__ out, const uint32_t* __restrict__ rows0, uint32_t mask0,
                              const uint32_t* __restrict__ rows1, uint32_t mask1, const uint32_t* __restrict__ key_rest,
                              uint32_t words, uint32_t v, uint32_t flags) {
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x) {
        const uint32_t row = w / kSideWords;
        uint32_t x = 0;
        if ((mask0 >> row) & 1u) x ^= rows0[w];
        if ((mask1 >> row) & 1u) x ^= rows1[w];
        if ((flags & kXorFlag) && 32ull * w < v) x ^= __byte_perm(__ldg(key_rest + w), 0, 0x0123);
        out[w] = x;
    }
}

size_t row_words(int log_np) { return (size_t(1) << (log_np - kChunkLog)) * kSideWords; }

}  // namespace

ChunkPlan chunk_plan(const BlockGeom& g) {
    ChunkPlan p;
    p.side = kSide;
    p.rows = (g.out_bits + p.side - 1u) / p.side;
    p.cols = (uint32_t)(((uint64_t)g.h + 1u + p.side - 1u) / p.side);
    // A chunk transform's key has side + 1 positions, the last one otherwise zero: when the taps past the last
    // full column are exactly one (h = cols * side, e.g. v = 3n/8), that tap takes the last column's
    // spare position instead of a column of its own.  Its seed index (i - h) lies in the column's seed
    // window like every other tap's.
    if (p.cols > 1 && ((uint64_t)g.h + 1u) % p.side == 1u) p.cols -= 1;
    p.diagonals = p.rows + p.cols - 1u;
    return p;
}

// Row passes for every column and window spectra for every diagonal at v = 3n/8.
size_t chunk_units(int log_np) { return 3 * (size_t(1) << (log_np - kChunkLog - 1)) + 1; }

bool chunk_keeps(const ChunkPlan& p, uint32_t units) { return units >= p.cols + p.diagonals; }

size_t chunk_staging_words(int log_np) {
    return 2 * (3 * (size_t)kSideWords + row_words(log_np)) + 2 * (size_t)kSideWords + 64;
}

void chunk_staging(int log_np, uint32_t* st, unsigned long long* counts, uint32_t* planes0, ChunkBuffers* cb) {
    for (ChunkLane& L : cb->lane) {
        L.window = st;
        L.result = st + 2 * kSideWords;
        L.rows = st + 3 * kSideWords;
        st = L.rows + row_words(log_np);
        L.pairs = counts;
        counts += 2 * kChunkCols;
    }
    cb->lane[0].sc.planes = planes0;
    cb->lane[1].sc.planes = st;
    cb->key_cnt = counts;
    cb->seed_cnt = counts + kChunkCols;
}

int chunk_kernel_count(const BlockGeom& g) {
    const ChunkPlan p = chunk_plan(g);
    // window, bit rows, passes A and B, counts per diagonal; bit rows and pass A per column; passes B and C and finish
    // per chunk, and the XOR of all but a lane's first one of a row; the final words
    uint32_t n = 5u * p.diagonals + 2u * p.cols + 4u * p.rows * p.cols + 1u;
    for (uint32_t a = 0; a < p.rows; ++a) n -= std::min(2u, p.cols);  // a row's columns alternate between the lanes
    return (int)n;
}

int launch_chunked_block(const BlockGeom& g, const BlockGeom& gc, const uint32_t* seed, const uint32_t* key_start,
                         const uint32_t* key_rest, uint32_t flags, uint32_t* out_words, const ChunkBuffers& cb,
                         bool seed_ready, unsigned int* resid_bits, int num_sms, cudaStream_t s) {
    const ChunkPlan p = chunk_plan(g);
    const size_t N = size_t(1) << gc.log_n;
    const int rows = (int)p.rows, cols = (int)p.cols, held = std::min<int>(cols, (int)cb.count);
    const bool keep = chunk_keeps(p, cb.count);
    cudaError_t err = cudaMemsetAsync(resid_bits, 0, sizeof(unsigned int), s);
    if (err != cudaSuccess) return (int)err;
    int rc = 0;
    auto check = [&](cudaError_t e) {
        if (!rc) rc = (int)e;
    };
    auto fork = [&] {
        check(cudaEventRecord(cb.fork, s));
        check(cudaStreamWaitEvent(cb.lane[1].s, cb.fork, 0));
    };
    auto join = [&] {
        check(cudaEventRecord(cb.join, cb.lane[1].s));
        check(cudaStreamWaitEvent(s, cb.join, 0));
    };
    // Column b's row pass: key bits b side .. b side + side - 1, the last column's up to bit h.
    auto key_rows = [&](const ChunkLane& L, int b, float2* Y, unsigned long long* cnt) {
        BlockGeom gk = gc;
        const uint64_t first = (uint64_t)b * kSide;
        gk.h = b == cols - 1 ? (uint32_t)(g.h - first) : kSide - 1u;
        if (!rc) rc = launch_bit_rows(gk, key_start + first / 32u, false, L.sc.planes, L.s, kOneBlock, cnt);
        if (!rc) rc = launch_pass_a(gc, L.sc.planes, false, Y, cnt, num_sms, L.s);
    };
    fork();
    for (int b = 0; b < held; ++b) key_rows(cb.lane[b & 1], b, cb.units + (size_t)b * N, cb.key_cnt + b);
    join();  // both lanes' columns
    fork();
    uint32_t mask[2] = {0u, 0u};
    for (int d = -(cols - 1), turn = 0; d < rows && !rc; ++d, ++turn) {
        const ChunkLane& L = cb.lane[turn & 1];
        float2* const spec = keep ? cb.units + (size_t)(cols + turn) * N : L.spec;
        unsigned long long* const cnt = cb.seed_cnt + (keep ? turn : turn & 1);
        if (!seed_ready) {
            k_seed_window<<<2 * num_sms, 256, 0, L.s>>>(L.window, seed, g.n / 32u, d);
            check(cudaGetLastError());
            if (!rc) rc = launch_seed_spectrum(gc, L.window, spec, L.sc, cnt, num_sms, L.s);
        }
        k_chunk_counts<<<1, cols, 0, L.s>>>(L.pairs, cb.key_cnt, cnt, held);
        check(cudaGetLastError());
        for (int a = std::max(0, d); a < std::min(rows, cols + d) && !rc; ++a) {
            const int b = a - d;
            const bool first = !((mask[turn & 1] >> a) & 1u);
            mask[turn & 1] |= 1u << a;
            BlockGeom gr = gc;
            gr.out_bits = (uint32_t)std::min<uint64_t>(kSide, g.out_bits - (uint64_t)a * kSide);
            float2* const Y = b < held ? cb.units + (size_t)b * N : L.sc.work;
            if (b >= held) key_rows(L, b, Y, L.pairs + 2 * b);
            uint32_t* const row = L.rows + (size_t)a * kSideWords;
            if (!rc)
                rc = launch_pass_b(gc, false, b < held ? cb.unit_maps[b] : *L.sc.maps, Y, L.sc.work2, spec, L.sc.err,
                                   num_sms, L.s);
            if (!rc)
                rc = launch_pass_c(gr, *L.sc.maps, L.sc.work2, L.pairs + 2 * b, L.sc.planes, resid_bits, L.sc.err, num_sms,
                                   L.s);
            if (!rc) rc = launch_finish(gr, L.sc.planes, nullptr, 0u, first ? row : L.result, L.s);
            if (!first && !rc) {
                k_xor_rows<<<2 * num_sms, 256, 0, L.s>>>(reinterpret_cast<uint4*>(row),
                                                         reinterpret_cast<const uint4*>(L.result),
                                                         (gr.out_bits + 127u) / 128u);
                check(cudaGetLastError());
            }
        }
    }
    join();
    if (rc) return rc;
    k_chunk_final<<<4 * num_sms, 256, 0, s>>>(out_words, cb.lane[0].rows, mask[0], cb.lane[1].rows, mask[1], key_rest,
                                              (g.out_bits + 31u) / 32u, g.v, flags);
    return (int)cudaGetLastError();
}

}  // namespace pa
