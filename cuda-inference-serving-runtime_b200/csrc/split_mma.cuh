// Float products of 64 x 64 tiles on the tensor cores (mma.sync m16n8k16, bfloat16 operands, float sums).
//
// A float is three bfloat16: x = b0 + b1 + b2 with b0 = x rounded, b1 = (x - b0) rounded, b2 the rest.  Both subtractions
// are exact and 3 x 8 bits hold a float's 24, so nothing of x is lost (but below about 2^-110, where the parts run out of
// exponents).  Of the nine products of parts the six largest are taken; what is left out is 2^-24 of the product and less, a
// float's own rounding.  The split of a float into bfloat16 parts for products is Henry, Tang and Heinecke's ("Leveraging the
// bfloat16 artificial intelligence datatype for higher-precision computations", 2019).
//
// Infinities, NaN and floats that round to a bfloat16 infinity have NaN among their parts, and zeros times those reach results
// that hold nothing of the number.  Every result that such a number touches is NaN, so a kernel looks at its sums at the end
// (not_finite) and, where any thread of the CTA has found one, makes its pass once more with PLAIN tiles and products: these
// hold a float's bits and use float multiply-adds.  That pass is a function of its own, never inlined: the registers of the
// usual one stay as they are.
//
// The float recurrences use it for their chunk products, which on the CUDA cores ran at a fifth of the multiply-add rate:
// a thread's 8 x 4 tile there loads twelve 16-byte words per 128 multiply-adds and waits for them.  Measured on a B200: this
// instruction runs at 548 TFLOP/s, so six of them at 91, where float multiply-adds without dependences reach 69.
// Error of a recurrence's outputs against 64 bits, 64 to 2048 tokens: 1.1e-7 with these products, 1.3e-7 to 2.2e-7 with
// chains of float multiply-adds.
#pragma once
#include "common.cuh"

namespace {
constexpr int SPLIT_LD = 72;          // row stride of a plane: 144 bytes, eight neighbouring rows in different banks
struct SplitTile { __nv_bfloat16 part[3][64][SPLIT_LD]; };     // 27,648 bytes

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// the three parts of two floats, packed (x in the low half)
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&p)[3]) {
    p[0] = bf16_pair(x, y);
    x -= __uint_as_float(p[0] << 16); y -= __uint_as_float(p[0] & 0xffff0000u);
    p[1] = bf16_pair(x, y);
    x -= __uint_as_float(p[1] << 16); y -= __uint_as_float(p[1] & 0xffff0000u);
    p[2] = bf16_pair(x, y);
}
// Results that parts may not have carried: those that are not finite, and those other than zero below 2^-64.  Of several, the largest oddness tells whether
// there is one: from ODD on.
constexpr uint32_t ODD = 0x7f800000u - 0x1f800000u;
__device__ __forceinline__ uint32_t oddness(float x) {
    const uint32_t size = __float_as_uint(x) & 0x7fffffffu;
    return size ? size - 0x1f800000u : 0u;         // below 2^-64: around to the largest numbers
}
// PLAIN: the upper and the lower halves of the floats' bits in the first two parts, zeros in the third
template <bool PLAIN>
__device__ __forceinline__ void tile_pair(float x, float y, uint32_t (&p)[3]) {
    if (!PLAIN) return split_pair(x, y, p);
    const uint32_t a = __float_as_uint(x), b = __float_as_uint(y);
    p[0] = (a >> 16) | (b & 0xffff0000u); p[1] = (a & 0xffffu) | (b << 16); p[2] = 0u;
}
template <bool PLAIN>
__device__ __forceinline__ void tile_store2(SplitTile& t, int row, int col, float x, float y) {       // col even
    uint32_t p[3];
    tile_pair<PLAIN>(x, y, p);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&t.part[i][row][col]) = p[i];
}
template <bool PLAIN>
__device__ __forceinline__ void tile_store4(SplitTile& t, int row, int col, float4 v) {       // col a multiple of 4
    uint32_t a[3], b[3];
    tile_pair<PLAIN>(v.x, v.y, a);
    tile_pair<PLAIN>(v.z, v.w, b);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(&t.part[i][row][col]) = make_uint2(a[i], b[i]);
}
template <bool PLAIN>
__device__ __forceinline__ float tile_value(const SplitTile& t, int row, int col) {
    if (PLAIN) return __uint_as_float(((uint32_t)__bfloat16_as_ushort(t.part[0][row][col]) << 16) | __bfloat16_as_ushort(t.part[1][row][col]));
    return to_float(t.part[0][row][col]) + (to_float(t.part[1][row][col]) + to_float(t.part[2][row][col]));
}
// eight neighbouring floats of a tile's row put together again (col a multiple of 8)
template <bool PLAIN>
__device__ __forceinline__ void tile_read8(const SplitTile& t, int row, int col, float (&v)[8]) {
    if (PLAIN) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = tile_value<true>(t, row, col + j);
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll
    for (int i = 2; i >= 0; --i) {
        const uint4 w = *reinterpret_cast<const uint4*>(&t.part[i][row][col]);
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { v[2 * j] += __uint_as_float(u[j] << 16); v[2 * j + 1] += __uint_as_float(u[j] & 0xffff0000u); }
    }
}

template <bool TRANS>
__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], const __nv_bfloat16* p) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(p);
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
    else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc (rows m0 .. m0 + 15, columns n0 .. n0 + 31 of the product) += A B over k in [0, 16 steps).  A is stored [m][k], or
// [k][m] with A_KM; B [n][k], or [k][n] with B_KN.  All lanes of a warp.  A thread's acc[j] holds rows m0 + lane / 4 (+ 8
// for elements 2 and 3) and columns n0 + 8 j + 2 (lane % 4) and the next.
// The tensor core cuts a sum instead of rounding it, so it sums sixteen terms at a time, from zero and the smallest parts
// first, and the sums of sixteen are added with rounding: four roundings for 64 terms, where a chain of float multiply-adds
// has 64.  A warp has a 16 x 32 part: with 32 x 32 the registers left twelve warps on an SM and every instruction waited (a
// third of the issue slots used).
template <bool A_KM, bool B_KN>
__device__ __forceinline__ void split_product(float (&acc)[4][4], const SplitTile& A, const SplitTile& B, int m0, int n0, int steps) {
    const int lane = threadIdx.x & 31, l7 = lane & 7, lo = (lane >> 3) & 1, hi = lane >> 4;
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        const int k = 16 * s;
        uint32_t a[3][4], b[3][2][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            load_matrices<A_KM>(a[p], A_KM ? &A.part[p][k + l7 + 8 * hi][m0 + 8 * lo] : &A.part[p][m0 + l7 + 8 * lo][k + 8 * hi]);
#pragma unroll
            for (int j = 0; j < 2; ++j)
                load_matrices<B_KN>(b[p][j], B_KN ? &B.part[p][k + l7 + 8 * lo][n0 + 16 * j + 8 * hi] : &B.part[p][n0 + 16 * j + l7 + 8 * hi][k + 8 * lo]);
        }
        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
        float t[4][4] = {};
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_bf16(t[j], a[PA[q]], b[PB[q]][j >> 1][2 * (j & 1)], b[PB[q]][j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[j][e] += t[j][e];
    }
}

// The same elements from tiles that hold floats, by multiply-adds in the order of k.  LOWER: A holds nothing right of its
// diagonal, and what B has there is left out.
template <bool A_KM, bool B_KN, bool LOWER>
__device__ __forceinline__ void plain_product(float (&acc)[4][4], const SplitTile& A, const SplitTile& B, int m0, int n0, int steps) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int m = m0 + 8 * half + (lane >> 2), last = LOWER ? min(16 * steps - 1, m) : 16 * steps - 1;
#pragma unroll 1
        for (int k = 0; k <= last; ++k) {
            const float a = A_KM ? tile_value<true>(A, k, m) : tile_value<true>(A, m, k);
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int n = n0 + 8 * j + 2 * (lane & 3) + e;
                    acc[j][2 * half + e] = fmaf(a, B_KN ? tile_value<true>(B, k, n) : tile_value<true>(B, n, k), acc[j][2 * half + e]);
                }
        }
    }
}
template <bool PLAIN, bool A_KM, bool B_KN, bool LOWER = false>
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const SplitTile& A, const SplitTile& B, int m0, int n0, int steps) {
    if (PLAIN) plain_product<A_KM, B_KN, LOWER>(acc, A, B, m0, n0, steps);
    else split_product<A_KM, B_KN>(acc, A, B, m0, n0, steps);
}
__device__ __forceinline__ int not_finite(const float (&acc)[4][4]) {
    float z = 0.f;                        // 0 x finite is 0, else NaN, and a NaN stays
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) z = fmaf(acc[j][e], 0.f, z);
    return z != 0.f;
}
}  // namespace
