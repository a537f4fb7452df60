// inverse.cuh -- modular inverses of BN254 field elements by divsteps.
//
// The division steps of Bernstein and Yang ("Fast constant-time gcd
// computation and modular inversion", CHES 2019),
//   delta > 0, g odd:  (delta, f, g) <- (1 - delta, g, (g - f) / 2)
//   otherwise:         (delta, f, g) <- (1 + delta, f, (g + (g mod 2) f) / 2),
// from f = p, g = a until g = 0, when f = +-1.  They start at delta = 1/2
// instead of the paper's 1; that variant, and its bound of 590 steps for
// operands below 2^256, are from P. Wuille's "safegcd-bounds"
// (github.com/sipa/safegcd-bounds, 2021).  The same steps modulo p take (0, 1)
// to (d, e) with f = d a and g = e a mod p throughout, so that a^-1 = f d.
//
// S = 30 steps depend on the low S bits of f and g alone, so they run on two
// registers and leave a matrix T, (f, g) <- T (f, g) / 2^S, whose rows have
// |x| + |y| <= 2^S: each step at most doubles the larger row.  All numbers are
// 32-bit words in two's complement, and the matrix is applied to them without
// signs: with x' = x + 2^S, y' = y + 2^S, both in [0, 2^(S+1)],
//   (x f + y g) / 2^S = (x' f + y' g) / 2^S - (f + g),
// one f + g for both rows.  x' + y' <= 3 2^S, so that x' f_i + y' g_i + m p_i
// and a carry fit 64 bits for any words and m < 2^S: with S = 31 they would not.
// f and g stay below p in magnitude.  To d and e a multiple m p is added that
// makes the low S bits vanish, which moves them by less than p a round: after R
// rounds |d| <= 1 + R p, and nothing is reduced before the end.
//
// Bound by the latency of its dependent steps where one point is converted:
// R = 20 rounds of 30 dependent steps, against the 254 dependent squarings
// and about 130 products of a Fermat power.  Measured on one point: an MSM with
// its affine conversion 1063 -> 881 us (1000 points); a proof with its wire
// form (one warp a point) 2963 -> 2358 us (2^12 constraints).
#pragma once
#include <cstdint>

namespace lzk {

constexpr int kInvStepBits = 30, kInvRounds = 20;
static_assert(kInvStepBits * kInvRounds >= 590, "too few steps for some operands");

// Nine 32-bit words, two's complement: 2^254 moduli times a few dozen.
struct Int9 {
    uint32_t w[9];
    __host__ __device__ __forceinline__ uint32_t sign() const { return (uint32_t)((int32_t)w[8] >> 31); }
};
__host__ __device__ __forceinline__ Int9 operator+(const Int9& a, const Int9& b)
{
    Int9 r;
#ifdef __CUDA_ARCH__
    asm("add.cc.u32  %0, %9,  %18;\n\t"
        "addc.cc.u32 %1, %10, %19;\n\t"
        "addc.cc.u32 %2, %11, %20;\n\t"
        "addc.cc.u32 %3, %12, %21;\n\t"
        "addc.cc.u32 %4, %13, %22;\n\t"
        "addc.cc.u32 %5, %14, %23;\n\t"
        "addc.cc.u32 %6, %15, %24;\n\t"
        "addc.cc.u32 %7, %16, %25;\n\t"
        "addc.u32    %8, %17, %26;"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7]), "=r"(r.w[8])
        : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]), "r"(a.w[8]),
          "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]), "r"(b.w[8]));
#else
    uint64_t c = 0;
    for (int i = 0; i < 9; i++, c >>= 32) r.w[i] = (uint32_t)(c += (uint64_t)a.w[i] + b.w[i]);
#endif
    return r;
}
__host__ __device__ __forceinline__ Int9 operator-(const Int9& a, const Int9& b)
{
    Int9 r;
#ifdef __CUDA_ARCH__
    asm("sub.cc.u32  %0, %9,  %18;\n\t"
        "subc.cc.u32 %1, %10, %19;\n\t"
        "subc.cc.u32 %2, %11, %20;\n\t"
        "subc.cc.u32 %3, %12, %21;\n\t"
        "subc.cc.u32 %4, %13, %22;\n\t"
        "subc.cc.u32 %5, %14, %23;\n\t"
        "subc.cc.u32 %6, %15, %24;\n\t"
        "subc.cc.u32 %7, %16, %25;\n\t"
        "subc.u32    %8, %17, %26;"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7]), "=r"(r.w[8])
        : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]), "r"(a.w[8]),
          "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]), "r"(b.w[8]));
#else
    uint64_t c = 1;
    for (int i = 0; i < 9; i++, c >>= 32) r.w[i] = (uint32_t)(c += (uint64_t)a.w[i] + (uint32_t)~b.w[i]);
#endif
    return r;
}
// p 2^k
template <class P>
__host__ __device__ __forceinline__ Int9 shifted_modulus(int k)
{
    Int9 r;
    _Pragma("unroll") for (int i = 0; i < 9; i++)
        r.w[i] = (i < 8 ? P::p(i) << k : 0u) | (i && k ? P::p(i - 1) >> (32 - k) : 0u);
    return r;
}

// The matrix of S steps, biased by 2^S.
struct StepMatrix {
    uint32_t ff, fg, gf, gg;   // f <- (ff f + fg g) / 2^S, g <- (gf f + gg g) / 2^S
};

// S steps on the low words f (odd) and g; half holds delta - 1/2.  Every step
// is the same branch-free code, so the lanes of a warp stay together: a
// version that skips runs of zero bits took more instructions per warp, since
// the slowest lane sets its length.
__host__ __device__ __forceinline__ StepMatrix divsteps(int32_t& half, uint32_t f, uint32_t g)
{
    uint32_t ff = 1, fg = 0, gf = 0, gg = 1;
    _Pragma("unroll 6") for (int i = 0; i < kInvStepBits; i++) {
        const uint32_t odd = g & 1u, swap = (0u - odd) & ~(uint32_t)(half >> 31);   // all ones: f takes g
        const uint32_t k = odd | swap;                                              // g takes g + k f: k = 0, 1 or -1
        const uint32_t g1 = g + k * f, gf1 = gf + k * ff, gg1 = gg + k * fg;
        f = (g & swap) | (f & ~swap);
        ff = ((gf & swap) | (ff & ~swap)) << 1;
        fg = ((gg & swap) | (fg & ~swap)) << 1;
        g = g1 >> 1;
        gf = gf1;
        gg = gg1;
        half = (int32_t)(((uint32_t)half ^ swap) + 1u);   // -half or half + 1
    }
    constexpr uint32_t bias = 1u << kInvStepBits;
    return {ff + bias, fg + bias, gf + bias, gg + bias};
}

// (x a + y b) / 2^S - sum for a biased row (x, y) and sum = a + b: the row
// without its bias.  MOD: plus the multiple of p that makes it whole (the row
// of f and g is whole by itself).
template <class P, bool MOD>
__host__ __device__ __forceinline__ Int9 apply_row(uint32_t x, uint32_t y, const Int9& a, const Int9& b, const Int9& sum)
{
    uint64_t acc = (uint64_t)x * a.w[0] + (uint64_t)y * b.w[0];
    uint32_t m = 0;
    if (MOD) {
        m = ((uint32_t)acc * P::INV) & ((1u << kInvStepBits) - 1);   // INV = -1 / p mod 2^32
        acc += (uint64_t)m * P::p(0);
    }
    uint32_t last = (uint32_t)acc;
    Int9 q;
    _Pragma("unroll") for (int i = 1; i < 10; i++) {
        uint32_t t;
        acc >>= 32;
        if (i < 9) {
            acc += (uint64_t)x * a.w[i < 9 ? i : 0];
            acc += (uint64_t)y * b.w[i < 9 ? i : 0];
            if (MOD && i < 8) acc += (uint64_t)m * P::p(i < 8 ? i : 0);
            t = (uint32_t)acc;
        } else {
            t = (uint32_t)acc - (a.sign() & x) - (b.sign() & y);   // the words above a negative operand's nine
        }
        q.w[i - 1] = last >> kInvStepBits | t << (32 - kInvStepBits);
        last = t;
    }
    return q - sum;
}

// a^-1 mod p of an integer a < p given as 8 words (0 for a = 0)
template <class P>
__host__ __device__ __forceinline__ void inverse_int(uint32_t out[8], const uint32_t a[8])
{
    Int9 f = shifted_modulus<P>(0), g, d, e;
    _Pragma("unroll") for (int i = 0; i < 9; i++) {
        g.w[i] = i < 8 ? a[i < 8 ? i : 0] : 0u;
        d.w[i] = 0;
        e.w[i] = i == 0;
    }
    int32_t half = 0;
    _Pragma("unroll 1") for (int round = 0; round < kInvRounds; round++) {
        uint32_t any = 0;
        _Pragma("unroll") for (int i = 0; i < 9; i++) any |= g.w[i];
        if (any == 0) break;
        const StepMatrix T = divsteps(half, f.w[0], g.w[0]);
        const Int9 fg = f + g, de = d + e;
        const Int9 f1 = apply_row<P, false>(T.ff, T.fg, f, g, fg), d1 = apply_row<P, true>(T.ff, T.fg, d, e, de);
        g = apply_row<P, false>(T.gf, T.gg, f, g, fg);
        e = apply_row<P, true>(T.gf, T.gg, d, e, de);
        f = f1;
        d = d1;
    }
    // f d with f = +-1 and |d| <= 1 + 20 p, plus 32 p if negative, modulo p
    const uint32_t flip = f.sign();
    Int9 r;
    _Pragma("unroll") for (int i = 0; i < 9; i++) r.w[i] = flip;
    _Pragma("unroll") for (int i = 0; i < 9; i++) d.w[i] ^= flip;
    r = d - r;
    const uint32_t negative = r.sign();
    Int9 up = shifted_modulus<P>(5);
    _Pragma("unroll") for (int i = 0; i < 9; i++) up.w[i] &= negative;
    r = r + up;
    static_assert(kInvRounds + 1 < 32, "the range the subtractions below start from");
    _Pragma("unroll") for (int k = 4; k >= 0; k--) {
        const Int9 t = r - shifted_modulus<P>(k);
        const uint32_t keep = t.sign();
        _Pragma("unroll") for (int i = 0; i < 9; i++) r.w[i] = (r.w[i] & keep) | (t.w[i] & ~keep);
    }
    _Pragma("unroll") for (int i = 0; i < 8; i++) out[i] = r.w[i];
}

}  // namespace lzk
