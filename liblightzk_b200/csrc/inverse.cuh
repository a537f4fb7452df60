// inverse.cuh -- modular inverses of BN254 field elements by divsteps.
//
// The greatest-common-divisor iteration of Bernstein and Yang ("Fast
// constant-time gcd computation and modular inversion", CHES 2019) in its
// half-delta form, which needs at most 590 divsteps for 256-bit operands:
//   delta > 0, g odd:  (delta, f, g) <- (1 - delta, g, (g - f) / 2)
//   otherwise:         (delta, f, g) <- (1 + delta, f, (g + (g mod 2) f) / 2)
// from delta = 1/2, f = p, g = a, until g = 0; then f = +-1 and a^-1 follows
// from the same steps applied to (0, 1) modulo p.
//
// 30 steps at a time depend only on the low 30 bits of f and g, so they run
// on single registers and leave a 2 x 2 matrix of signed 31-bit entries that
// is then applied to the full numbers (nine signed 30-bit limbs).  Inside the
// 30 steps, runs of zero bits are taken at once, and while delta < 0 (f stays)
// up to six bits of g are cleared by one multiple of f.
//
// Bound by the latency of its dependent steps where one point is converted:
// 20 rounds of about 350 instructions here, against the 254 dependent
// squarings and about 130 products of a Fermat power.  Measured on one point:
// the affine conversion 228 -> 46 us (G1); the three points of a proof's wire
// form, one warp each, 686 -> 80 us.
#pragma once
#include <cstdint>

namespace lzk {

constexpr int32_t kM30 = 0x3fffffff;

// 30-bit limb i of the modulus
template <class P>
__host__ __device__ constexpr int32_t p30(int i)
{
    const int b = 30 * i, w = b / 32, s = b % 32;
    const uint64_t lo = P::p(w), hi = w + 1 < 8 ? P::p(w + 1) : 0u;
    return (int32_t)(((lo | hi << 32) >> s) & (uint64_t)kM30);
}

struct Divsteps30 {
    int32_t u, v, q, r;   // 2^30 f' = u f + v g, 2^30 g' = q f + r g
};

// 30 divsteps on the low words f0 (odd), g0; d holds delta - 1/2
__host__ __device__ __forceinline__ void divsteps30(int32_t& d, uint32_t f, uint32_t g, Divsteps30& t)
{
    int32_t u = 1, v = 0, q = 0, r = 1;
    int rem = 30;
    for (;;) {
        const uint32_t stop = g | (0xffffffffu << rem);
#ifdef __CUDA_ARCH__
        const int z = __ffs((int)stop) - 1;
#else
        const int z = __builtin_ctz(stop);
#endif
        g >>= z;
        u = (int32_t)((uint32_t)u << z);
        v = (int32_t)((uint32_t)v << z);
        d += z;
        rem -= z;
        if (rem == 0) break;
        if (d >= 0) {
            uint32_t x = f; f = g; g = 0u - x;
            int32_t y = u; u = q; q = -y;
            y = v; v = r; r = -y;
            d = -d - 1;
        }
        // f stays for the next -d steps: w = -g / f mod 2^lim clears their
        // low bits (f (f^2 - 2) is -1/f modulo 64 for odd f)
        int lim = rem < -d ? rem : -d;
        if (lim > 6) lim = 6;
        const uint32_t w = (g * f * (f * f - 2u)) & ((1u << lim) - 1u);
        g += f * w;
        q = (int32_t)((uint32_t)q + (uint32_t)u * w);
        r = (int32_t)((uint32_t)r + (uint32_t)v * w);
    }
    t.u = u; t.v = v; t.q = q; t.r = r;
}

// a^-1 mod p of an integer a < p given as 8 limbs (0 for a = 0)
template <class P>
__host__ __device__ __forceinline__ void inverse_int(uint32_t out[8], const uint32_t a[8])
{
    int32_t f[9], g[9], d[9], e[9];
    _Pragma("unroll") for (int i = 0; i < 9; i++) {
        const int b = 30 * i, w = b / 32, s = b % 32;
        const uint64_t lo = a[w], hi = w + 1 < 8 ? a[w + 1] : 0u;
        f[i] = p30<P>(i);
        g[i] = (int32_t)(((lo | hi << 32) >> s) & (uint64_t)kM30);
        d[i] = 0;
        e[i] = i == 0;
    }
    const uint32_t pinv = 0u - P::INV;   // p^-1 mod 2^32
    int32_t delta = 0;
    _Pragma("unroll 1") for (int it = 0; it < 20; it++) {
        uint32_t any = 0;
        _Pragma("unroll") for (int i = 0; i < 9; i++) any |= (uint32_t)g[i];
        if (any == 0) break;
        Divsteps30 t;
        divsteps30(delta, (uint32_t)f[0] | (uint32_t)f[1] << 30, (uint32_t)g[0] | (uint32_t)g[1] << 30, t);
        const int64_t u = t.u, v = t.v, q = t.q, r = t.r;
        // (d, e) <- (u d + v e, q d + r e) / 2^30 mod p, kept in (-2p, p): a
        // negative operand counts as itself plus p
        const int32_t sd = d[8] >> 31, se = e[8] >> 31;
        int32_t md = (t.u & sd) + (t.v & se), me = (t.q & sd) + (t.r & se);
        int64_t cd = u * d[0] + v * e[0], ce = q * d[0] + r * e[0];
        md -= (int32_t)((pinv * (uint32_t)cd + (uint32_t)md) & (uint32_t)kM30);
        me -= (int32_t)((pinv * (uint32_t)ce + (uint32_t)me) & (uint32_t)kM30);
        cd = (cd + (int64_t)p30<P>(0) * md) >> 30;
        ce = (ce + (int64_t)p30<P>(0) * me) >> 30;
        int64_t cf = (u * f[0] + v * g[0]) >> 30, cg = (q * f[0] + r * g[0]) >> 30;
        _Pragma("unroll") for (int i = 1; i < 9; i++) {
            cd += u * d[i] + v * e[i] + (int64_t)p30<P>(i) * md;
            ce += q * d[i] + r * e[i] + (int64_t)p30<P>(i) * me;
            cf += u * f[i] + v * g[i];
            cg += q * f[i] + r * g[i];
            d[i - 1] = (int32_t)cd & kM30; cd >>= 30;
            e[i - 1] = (int32_t)ce & kM30; ce >>= 30;
            f[i - 1] = (int32_t)cf & kM30; cf >>= 30;
            g[i - 1] = (int32_t)cg & kM30; cg >>= 30;
        }
        d[8] = (int32_t)cd; e[8] = (int32_t)ce; f[8] = (int32_t)cf; g[8] = (int32_t)cg;
    }
    // a^-1 = f d mod p with f = +-1, d in (-2p, p)
    const int32_t neg = f[8] >> 31;
    int32_t add = d[8] >> 31;
    _Pragma("unroll") for (int i = 0; i < 9; i++) d[i] = ((d[i] + (p30<P>(i) & add)) ^ neg) - neg;
    _Pragma("unroll") for (int i = 0; i < 8; i++) { d[i + 1] += d[i] >> 30; d[i] &= kM30; }
    add = d[8] >> 31;
    _Pragma("unroll") for (int i = 0; i < 9; i++) d[i] += p30<P>(i) & add;
    _Pragma("unroll") for (int i = 0; i < 8; i++) { d[i + 1] += d[i] >> 30; d[i] &= kM30; }
    _Pragma("unroll") for (int i = 0; i < 8; i++) {
        const int l = 32 * i / 30, s = 32 * i % 30;   // 32-bit word i starts inside limb l
        uint64_t x = (uint64_t)(uint32_t)d[l] >> s;
        x |= (uint64_t)(uint32_t)d[l + 1] << (30 - s);
        if (l + 2 < 9) x |= (uint64_t)(uint32_t)d[l + 2] << (60 - s);
        out[i] = (uint32_t)x;
    }
}

}  // namespace lzk
