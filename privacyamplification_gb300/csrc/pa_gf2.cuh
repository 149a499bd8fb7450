// pa_gf2.cuh -- bit-sliced arithmetic in GF(2^32) for the exact path (pa_exact.cu).
//
// Elements are written in the tower basis of the nimbers (Conway, On Numbers and Games, ch. 6):
// GF(2^(2h)) = GF(2^h)[X] / (X^2 + X + 2^(h-1)), so element bits 0 .. h-1 and h .. 2h-1 are the two GF(2^h)
// coefficients, every GF(2^(2^k)) is the elements below 2^(2^k), and the trace to GF(2) is the top bit.
// Bit-sliced: an element vector is K words, word c holding bit c of 32 elements, one per lane bit.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pa {
namespace gf2 {

// ------------------------------------------------------------------------ constants, at compile time
// Product of two elements below 2^(2^k).
__host__ __device__ constexpr uint32_t nim_mul(uint32_t a, uint32_t b, int k = 5) {
    if (!a || !b) return 0;
    if (k == 0) return a & b;
    const int h = 1 << (k - 1);
    const uint32_t m = (1u << h) - 1u;
    const uint32_t a0 = a & m, a1 = a >> h, b0 = b & m, b1 = b >> h;
    const uint32_t p0 = nim_mul(a0, b0, k - 1), p1 = nim_mul(a1, b1, k - 1);
    const uint32_t p2 = nim_mul(a0 ^ a1, b0 ^ b1, k - 1);
    return ((p2 ^ p0) << h) | (p0 ^ nim_mul(p1, 1u << (h - 1), k - 1));
}

// A Cantor basis: kCantor[0] = 1, kCantor[i]^2 + kCantor[i] = kCantor[i-1].  The subspace polynomials are then
// s_i(x) = s_{i-1}(x)^2 + s_{i-1}(x) with s_i(kCantor[j]) = kCantor[j - i], s_{2^k}(x) = x^(2^(2^k)) + x, and
// kCantor[0 .. 2^k - 1] spans GF(2^(2^k)).
constexpr uint32_t kCantor[32] = {
    0x1,       0x2,       0x4,       0xa,       0x14,       0x20,       0x4c,       0xae,
    0x152,     0x22e,     0x480,     0xa4c,     0x14fa,     0x2002,     0x4c32,     0xae98,
    0x15214,   0x22e7a,   0x48066,   0xa4cc0,   0x14fa06,   0x2002ba,   0x4c3284,   0xae98d4,
    0x15294e0, 0x22eba22, 0x480d6c2, 0xa4cd0b0, 0x14fa3b2a, 0x20027c50, 0x4c325d7a, 0xae986cfa};
constexpr bool cantor_ok() {
    if (kCantor[0] != 1u) return false;
    for (int i = 1; i < 32; ++i)
        if ((nim_mul(kCantor[i], kCantor[i]) ^ kCantor[i]) != kCantor[i - 1]) return false;
    return true;
}
static_assert(cantor_ok(), "kCantor is a Cantor basis");

// The field element z that a 16-bit segment's polynomial variable stands for; 1, z .. z^31 are a basis, so
// the product of two segments (degree <= 30) keeps its coefficients.
constexpr uint32_t kZ = 1u << 16;
struct Matrix {
    uint32_t row[32];
};
constexpr Matrix z_powers() {  // row[j] = z^j
    Matrix m{};
    m.row[0] = 1;
    for (int j = 1; j < 32; ++j) m.row[j] = nim_mul(m.row[j - 1], kZ);
    return m;
}
// Coordinates with respect to the trace form: row j, bit c = Tr(2^c z^j), so Tr(w z^j) is the parity of
// w & row[j].
constexpr Matrix dual_rows() {
    Matrix m{};
    const Matrix z = z_powers();
    for (int j = 0; j < 32; ++j)
        for (int c = 0; c < 32; ++c) m.row[j] |= (nim_mul(1u << c, z.row[j]) >> 31) << c;
    return m;
}
// Inverse of dual_rows(): row c, bit j -- the element whose traces against z^j are given bits.
constexpr Matrix dual_inverse() {
    Matrix a = dual_rows(), b{};
    for (int j = 0; j < 32; ++j) b.row[j] = 1u << j;
    for (int c = 0; c < 32; ++c) {
        int p = c;
        while (p < 32 && !((a.row[p] >> c) & 1u)) ++p;
        if (p == 32) return Matrix{};  // 1, z .. z^31 would be dependent
        const uint32_t ta = a.row[c], tb = b.row[c];
        a.row[c] = a.row[p];
        b.row[c] = b.row[p];
        a.row[p] = ta;
        b.row[p] = tb;
        for (int r = 0; r < 32; ++r)
            if (r != c && ((a.row[r] >> c) & 1u)) {
                a.row[r] ^= a.row[c];
                b.row[r] ^= b.row[c];
            }
    }
    return b;
}
constexpr Matrix transpose(const Matrix& m) {
    Matrix t{};
    for (int r = 0; r < 32; ++r)
        for (int c = 0; c < 32; ++c) t.row[c] |= ((m.row[r] >> c) & 1u) << r;
    return t;
}
constexpr Matrix kSegToField = transpose(z_powers());  // row c: which segment bits make field bit c
constexpr Matrix kTraceToField = dual_inverse();       // row c: which traces make field bit c
constexpr Matrix kFieldToTrace = dual_rows();          // row j: which field bits make trace j
static_assert(kTraceToField.row[0] != 0u, "1, z .. z^31 are independent");

// ------------------------------------------------------------------------ bit-sliced products
// x * 2^(K-1) in GF(2^K), the constant of the next tower step.
template <int K>
__host__ __device__ __forceinline__ void mul_g(const uint32_t (&x)[K], uint32_t (&y)[K]) {
    if constexpr (K == 1) {
        y[0] = x[0];
    } else {
        constexpr int H = K / 2;
        uint32_t lo[H], s[H], t[H];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            t[i] = x[H + i];
            s[i] = x[i] ^ x[H + i];
        }
        mul_g<H>(t, lo);
        mul_g<H>(lo, t);
        mul_g<H>(s, lo);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            y[i] = t[i];
            y[H + i] = lo[i];
        }
    }
}

// c = a b, bit-sliced, in GF(2^K): Karatsuba down the tower, four LOP3 per GF(4) product.
template <int K>
__host__ __device__ __forceinline__ void mul(const uint32_t (&a)[K], const uint32_t (&b)[K], uint32_t (&c)[K]) {
    if constexpr (K == 1) {
        c[0] = a[0] & b[0];
    } else if constexpr (K == 2) {
        const uint32_t p = a[1] & b[1];
        c[0] = (a[0] & b[0]) ^ p;
        c[1] = (a[1] & b[0]) ^ ((a[0] & b[1]) ^ p);
    } else {
        constexpr int H = K / 2;
        uint32_t x[H], y[H], p0[H], p1[H], p2[H];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            x[i] = a[H + i];
            y[i] = b[H + i];
        }
        mul<H>(x, y, p1);
        uint32_t u[H], w[H];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            u[i] = a[i];
            w[i] = b[i];
        }
        mul<H>(u, w, p0);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            x[i] ^= u[i];
            y[i] ^= w[i];
        }
        mul<H>(x, y, p2);
        mul_g<H>(p1, x);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            c[i] = p0[i] ^ x[i];
            c[H + i] = p2[i] ^ p0[i];
        }
    }
}

// Bit-sliced linear maps: out[r] = XOR of in[c] over the set bits c of the matrix's row r.
enum Map { kMapSegToField, kMapTraceToField, kMapFieldToTrace };
template <Map M, int ROWS, int COLS, int R = 0>
__host__ __device__ __forceinline__ void apply(const uint32_t (&in)[COLS], uint32_t (&out)[ROWS]) {
    if constexpr (R < ROWS) {
        constexpr uint32_t bits = M == kMapSegToField     ? kSegToField.row[R]
                                  : M == kMapTraceToField ? kTraceToField.row[R]
                                                          : kFieldToTrace.row[R];
        uint32_t v = 0;
#pragma unroll
        for (int c = 0; c < COLS; ++c)
            if ((bits >> c) & 1u) v ^= in[c];
        out[R] = v;
        apply<M, ROWS, COLS, R + 1>(in, out);
    }
}

}  // namespace gf2
}  // namespace pa
