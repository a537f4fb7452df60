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
// is then applied to the full numbers (nine signed 30-bit limbs).
//
// Bound by the latency of its dependent steps where one point is converted:
// 20 rounds of about 700 instructions here, against the 254 dependent
// squarings and about 130 products of a Fermat power.  Measured on one point:
// an MSM with its affine conversion 1063 -> 881 us (1000 points); a proof with
// its wire form (one warp a point) 2963 -> 2358 us (2^12 constraints).
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

// 30 divsteps on the low words f (odd), g; d holds delta - 1/2.  Every step
// is the same branch-free code, so the lanes of a warp stay together: a
// version that skips runs of zero bits took more instructions per warp, since
// the slowest lane sets its length.
__host__ __device__ __forceinline__ void divsteps30(int32_t& d, uint32_t f, uint32_t g, Divsteps30& t)
{
    uint32_t u = 1, v = 0, q = 0, r = 1;
    _Pragma("unroll 6") for (int i = 0; i < 30; i++) {
        const uint32_t bit = g & 1u, swap = (0u - bit) & ~(uint32_t)(d >> 31);   // all ones: swap f and g
        const uint32_t s = bit | swap;                                           // 0, 1 or -1
        const uint32_t ng = g + s * f, nq = q + s * u, nr = r + s * v;
        f = (g & swap) | (f & ~swap);
        u = ((q & swap) | (u & ~swap)) << 1;
        v = ((r & swap) | (v & ~swap)) << 1;
        g = ng >> 1;
        q = nq;
        r = nr;
        d = (int32_t)(((uint32_t)d ^ swap) + 1u);   // -d or d + 1
    }
    t.u = (int32_t)u; t.v = (int32_t)v; t.q = (int32_t)q; t.r = (int32_t)r;
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
