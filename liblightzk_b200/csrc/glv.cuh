// glv.cuh -- the endomorphism of BN254 G1 and the split of scalars over it
// (Gallant, Lambert and Vanstone, CRYPTO 2001).
//
// phi(x, y) = (beta x, y), beta a cube root of unity in Fq, is lambda (x, y)
// with lambda the matching cube root of unity in Fr (G1 has prime order, so
// this holds for every point).  A scalar k is written k1 + lambda k2 with
// |k1|, |k2| < 2^126: (k, 0) minus the nearest vector of the lattice of
// (a, b) with a + b lambda = 0 mod r, whose reduced basis is (-A, B), (-C, -A).
//   d1 = round(k A / r), d2 = round(k B / r),
//   k1 = k - d1 A - d2 C, k2 = d1 B - d2 A,
// with A / r and B / r as integers over 2^272.  The split is exact whatever
// the rounding; the bound holds with the error of the truncated constants.
//
// A product by a scalar, or the combination of an MSM's windows, then needs
// half the dependent doublings: the two halves run as separate points.
#pragma once
#include "field.cuh"

namespace lzk {

// beta, Montgomery form
__device__ __forceinline__ Fq glv_beta()
{
    return Fq{{0xd782e155u, 0x71930c11u, 0xffbe3323u, 0xa6bb947cu, 0xd4741444u, 0xaa303344u, 0x26594943u, 0x2c3b3f0du}};
}

constexpr uint32_t kGlvBits = 126;   // |k1|, |k2| < 2^kGlvBits

// t[0..NA+NB) = a b
template <int NA, int NB>
__host__ __device__ __forceinline__ void mul_words(uint32_t* t, const uint32_t* a, const uint32_t* b)
{
    _Pragma("unroll") for (int i = 0; i < NA + NB; i++) t[i] = 0;
    _Pragma("unroll") for (int i = 0; i < NB; i++) {
        uint32_t c = 0;
        _Pragma("unroll") for (int j = 0; j < NA; j++) {
            const uint64_t s = mac64(a[j], b[i], t[i + j], c);
            t[i + j] = (uint32_t)s;
            c = (uint32_t)(s >> 32);
        }
        t[i + NA] = c;
    }
}
// round(k g / 2^272) of the product's words: OUT words
template <int NG, int OUT>
__host__ __device__ __forceinline__ void mul_round272(uint32_t* d, const uint32_t k[8], const uint32_t* g)
{
    uint32_t t[8 + NG];
    mul_words<8, NG>(t, k, g);
    uint64_t s = (uint64_t)t[8] + 0x8000u;   // 2^271
    t[8] = (uint32_t)s;
    _Pragma("unroll") for (int i = 9; i < 8 + NG; i++) {
        s = (uint64_t)t[i] + (s >> 32);
        t[i] = (uint32_t)s;
    }
    _Pragma("unroll") for (int i = 0; i < OUT; i++)
        d[i] = t[8 + i] >> 16 | (9 + i < 8 + NG ? t[9 + i] << 16 : 0u);
}
// x -= y over 5 words
__host__ __device__ __forceinline__ void sub5(uint32_t x[5], const uint32_t* y)
{
    uint64_t b = 0;
    _Pragma("unroll") for (int i = 0; i < 5; i++) {
        const uint64_t s = (uint64_t)x[i] - y[i] - b;
        x[i] = (uint32_t)s;
        b = s >> 63;
    }
}
// two's complement x to its magnitude; true if it was negative
__host__ __device__ __forceinline__ bool magnitude(uint32_t out[4], const uint32_t x[5])
{
    const uint32_t m = 0u - (x[4] >> 31);
    uint64_t c = m & 1u;
    _Pragma("unroll") for (int i = 0; i < 4; i++) {
        c += (uint64_t)(x[i] ^ m);
        out[i] = (uint32_t)c;
        c >>= 32;
    }
    return m != 0;
}

// k = (-1)^n1 k1 + lambda (-1)^n2 k2 mod r for a canonical k < r
__host__ __device__ __forceinline__ void glv_split(const uint32_t k[8], uint32_t k1[4], bool& n1, uint32_t k2[4], bool& n2)
{
    const uint32_t A[2] = {0x94d213e3u, 0x89d32568u};
    const uint32_t B[4] = {0x7d4f1128u, 0x8211bbebu, 0xeeb859fcu, 0x6f4d8248u};
    const uint32_t C[4] = {0x1221250bu, 0x0be4e154u, 0xeeb859fdu, 0x6f4d8248u};
    const uint32_t gA[3] = {0xb3d76eb9u, 0x232ec7e0u, 0x0002d91du};
    const uint32_t gB[5] = {0xb18da5e3u, 0xd9d4391eu, 0xd2cf7a7bu, 0xf014a773u, 0x00024cceu};
    uint32_t d1[2], d2[4], t[8], x[5];
    mul_round272<3, 2>(d1, k, gA);
    mul_round272<5, 4>(d2, k, gB);
    _Pragma("unroll") for (int i = 0; i < 5; i++) x[i] = k[i];
    t[4] = 0;
    mul_words<2, 2>(t, d1, A);
    sub5(x, t);
    mul_words<4, 4>(t, d2, C);
    sub5(x, t);
    n1 = magnitude(k1, x);
    mul_words<4, 2>(t, B, d1);
    _Pragma("unroll") for (int i = 0; i < 5; i++) x[i] = t[i];
    mul_words<4, 2>(t, d2, A);
    sub5(x, t);
    n2 = magnitude(k2, x);
}

}  // namespace lzk
