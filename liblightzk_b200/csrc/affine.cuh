// affine.cuh -- bucket sums by rounds of batched affine additions.
//
// An XYZZ mixed addition costs 8 products and 2 squares; an affine addition
// costs a slope (1 product, given 1 / (x2 - x1)), a square and a product, plus
// its share of a batched inversion (Montgomery's trick: 3 products per element
// and one inversion per batch).  With the inverse by divsteps (inverse.cuh,
// about 25 products) and batches of tens of additions per thread, that is 5
// products, a square and a fraction, about two thirds of the mixed addition;
// for G2 the inversion runs on the norms, in Fq, and the addition costs a
// little over half.
//
// The sorted entries are laid out with every bucket starting at a multiple of
// 2^R slots (gaps hold kNoEntry), so pair j of a round is always slots 2j and
// 2j + 1 of one bucket, with no bucket bookkeeping: round 1 adds pairs of base
// points named by the entries, later rounds pairs of the round before's
// results, each leaving half as many points.  After R rounds a bucket of s
// entries holds ceil(s / 2^R) points, which the XYZZ accumulation finishes.
//
// A round is three launches over the same T threads, pairs j, j + T, ... to a
// thread (neighbouring threads touch neighbouring pairs): the running product
// of the thread's denominators, its prefixes parked in the output slots; the
// inverses of the threads' products, kInvGroup to an inversion; and, in the
// reverse order, slope and sum of each pair.  A pair with an infinity or of
// opposite points multiplies by one; equal points double.
//
// Products stay in the radix-2^52 form of field52.cuh between the loads and
// the stores (no packing to 8 x 32 bits, no conditional subtraction), with
// operands below 2p and results below 2p.  The plain product there is
// M(a, b) = a b / 2^260; the powers of two are settled once per batch by the
// constant that the inverse is multiplied with:
//   D_k = d_k 2^256 (Fq) or N_k = |d_k|^2 2^252 (norm of an Fq2 difference),
//   prefix_k = M(prefix_{k-1}, D_k),  inv_K = 2^518 / prefix_K, so that
//   M(inv_k, prefix_{k-1}) = 2^518 / D_k,  M(inv_k, D_k) = inv_{k-1},
// and a numerator n 2^256 times 2^518 / D_k gives 4 (n / d) 2^256, the slope
// scaled by 4: M(4L, 4L) = L^2 2^256 and M(4L, 4 w) = L w 2^256.
//
// Measured over a table, accumulation alone (G1 1000003 points, 15 M entries;
// G2 200003 points, 3.2 M): 2979 -> 2497 us and 1895 -> 1467 us.  A proof at
// 2^20 constraints, whose other work shares the GPU: 25.4 -> 20.8 ms.
//
// Bound by the issue of the products' FP64 and 64-bit integer instructions
// (about 2400 a G1 addition, against 4400 of an XYZZ mixed addition), round 1
// also by the gather of the bases, which it reads twice.  The kernels' code
// has to stay within the instruction cache: with every product inlined, or
// with the next round's prefixes formed in the sums' kernel, instruction
// fetches cost more than the work saved.
#pragma once
#include "msm.cuh"

namespace lzk {

struct D5 {
    double d[5];
};
struct L5 {
    uint64_t l[5];
};

__device__ __forceinline__ D5 to_d5(const uint64_t r[5])
{
    D5 x;
    _Pragma("unroll") for (int i = 0; i < 5; i++) x.d[i] = u52_to_d(r[i]);
    return x;
}
template <int S>
__device__ __forceinline__ D5 to_d5(const Fq& a)
{
    D5 x;
    to_d52<S>(x.d, a.v);
    return x;
}
// limbs (value < 2p) to the canonical element
__device__ __forceinline__ Fq canon52(const uint64_t r[5])
{
    uint32_t t[8];
    from_limbs52(t, r);
    return final_sub<FqP>(t);
}
// M(a, b) = a b / 2^260 mod p (limbs, < 2p) for a b < p 2^260, out of line
static __device__ __noinline__ L5 mont_call(const D5 a, const D5 b)
{
    L5 r;
    mont52_core<FqP>(r.l, a.d, b.d);
    return r;
}
static __device__ __noinline__ L5 mont_sqr_call(const D5 a)
{
    L5 r;
    mont52_sqr_core<FqP>(r.l, a.d);
    return r;
}
// two products, interleaved
struct L5x2 {
    L5 a, b;
};
static __device__ __noinline__ L5x2 mont2_call(const D5 a, const D5 b, const D5 c, const D5 d)
{
    L5x2 r;
    mont52_core<FqP>(r.a.l, a.d, b.d);
    mont52_core<FqP>(r.b.l, c.d, d.d);
    return r;
}
__device__ __forceinline__ D5 mont_d5(const D5& a, const D5& b) { return to_d5(mont_call(a, b).l); }
__device__ __forceinline__ Fq mont_fq(const D5& a, const D5& b) { return canon52(mont_call(a, b).l); }

// 2^260 mod p, the one of M
__device__ __forceinline__ L5 l5_one()
{
    return L5{{0x20880f6fce4b4ull, 0x49baa989a8455ull, 0x18f014a498908ull, 0x724f85a9201d8ull, 0x1f16424e1bb7ull}};
}
__device__ __forceinline__ D5 d5_one() { return to_d5(l5_one().l); }
// 2^518 / a for the a < 2p of these limbs: the integer inverse times 2^778
// under M
__device__ __forceinline__ L5 l5_inverse(const L5& a)
{
    Fq x = canon52(a.l);
    uint32_t y[8];
    inverse_int<FqP>(y, x.v);
    _Pragma("unroll") for (int i = 0; i < 8; i++) x.v[i] = y[i];
    const D5 c{{(double)0x8c91e0ff8e86aull, (double)0x25dab495b144full, (double)0xd80fe5cb1670aull,
                (double)0x61fd714e1c8e4ull, (double)0x43c5b7b6346ull}};
    return mont_call(to_d5<0>(x), c);
}

// a value below 2p parked in 32 bytes (one sector)
__device__ __forceinline__ void park(void* p, const L5& a)
{
    Fq t;
    from_limbs52(t.v, a.l);
    st_elem(static_cast<Fq*>(p), t);
}
__device__ __forceinline__ D5 unpark(const void* p) { return to_d5<0>(ld_elem(static_cast<const Fq*>(p))); }

// Operands of a round: entry v of the sorted list (FIRST), or the point
// src[v] of the round before.  load_x returns true for an infinity: a gap, a
// base at (0, 0), or a result with the marker.
template <bool FIRST, class F>
__device__ __forceinline__ bool load_x(const Aff<F>* src, uint32_t v, uint64_t nbases, F& x)
{
    if (FIRST) {
        if (v == kNoEntry) { x = F::zero(); return true; }
        const Aff<F>* b = src + (v & 0x7fffffffu);
        if (!LZK_CHECK((v & 0x7fffffffu) < nbases, 2)) { x = F::zero(); return true; }
        x = ldg_elem(&b->x);
        return x.is_zero() && ldg_elem(&b->y).is_zero();
    }
    x = ld_elem(&src[v].x);
    return is_marker(x);
}
template <bool FIRST, class F>
__device__ __forceinline__ F load_y(const Aff<F>* src, uint32_t v, uint64_t nbases)
{
    (void)nbases;
    if (FIRST) {
        if (v == kNoEntry || !LZK_CHECK((v & 0x7fffffffu) < nbases, 2)) return F::zero();
        F y = ldg_elem(&src[v & 0x7fffffffu].y);
        return v & 0x80000000u ? neg(y) : y;
    }
    return ld_elem(&src[v].y);
}

// Pair with equal x: the doubling's denominator 2 y and numerator 3 x^2, or
// ok = false for opposite points.
template <class F>
struct Doubling {
    F den, num;
    bool ok;
};
template <class F>
__device__ __noinline__ Doubling<F> same_x(const F x, const F y1, const F y2)
{
    Doubling<F> r;
    r.ok = y1 == y2 && !y1.is_zero();
    r.den = dbl(y1);
    F s = sqr(x);
    r.num = add(dbl(s), s);
    return r;
}

// The pairs of round r of a slice: slots [s0, s0 + slots) of the padded list
// below its total, halved r times.
template <class F>
__device__ __forceinline__ uint32_t round_pairs(const AffineRound<F>& a)
{
    const uint64_t t = *a.total;
    if (a.s0 >= t) return 0;
    return (uint32_t)((t - a.s0 < a.slots ? t - a.s0 : a.slots) >> a.r);
}
// the operands of pair j: two entries, or two of the last round's points
template <bool FIRST, class F>
__device__ __forceinline__ uint2 pair_at(const AffineRound<F>& a, uint32_t j)
{
    return FIRST ? __ldg(reinterpret_cast<const uint2*>(a.ent) + j) : make_uint2(2 * j, 2 * j + 1);
}

// The denominator of a pair, or one where its sum needs no addition.
template <bool FIRST>
__device__ __forceinline__ D5 pair_den(const Aff<Fq>* src, uint64_t nbases, uint2 v, const Fq& x1, const Fq& x2, bool skip)
{
    Fq d = sub_plus_p(x2, x1);
    if (!skip && x1 == x2) {
        const Doubling<Fq> e = same_x(x1, load_y<FIRST>(src, v.x, nbases), load_y<FIRST>(src, v.y, nbases));
        d = e.den;
        skip = !e.ok;
    }
    D5 D = to_d5<0>(d);
    if (skip) D = d5_one();
    return D;
}

template <bool FIRST>
__global__ void __launch_bounds__(kAffThreads, kAffBlocksG1) k_affine_prefix_g1(const AffineRound<Fq> a)
{
    const uint32_t np = round_pairs(a), T = gridDim.x * kAffThreads, t0 = blockIdx.x * kAffThreads + threadIdx.x;
    L5 acc = l5_one();
    for (uint32_t j = t0; j < np; j += T) {
        const uint2 v = pair_at<FIRST>(a, j);
        Fq x1, x2;
        bool skip = load_x<FIRST>(a.src, v.x, a.nbases, x1);
        skip |= load_x<FIRST>(a.src, v.y, a.nbases, x2);
        park(a.out + j, acc);
        const D5 D = pair_den<FIRST>(a.src, a.nbases, v, x1, x2, skip);
        mont52_core<FqP>(acc.l, to_d5(acc.l).d, D.d);
    }
    a.acc[t0] = acc;
}

// acc[t] <- 2^518 / acc[t] for t < count, kInvGroup to a thread
static __global__ void __launch_bounds__(kAffThreads) k_affine_invert(L5* __restrict__ acc, uint32_t count)
{
    const uint32_t T = gridDim.x * kAffThreads, t = blockIdx.x * kAffThreads + threadIdx.x;
    L5 a[kInvGroup], p[kInvGroup];
    _Pragma("unroll") for (int k = 0; k < kInvGroup; k++) {
        a[k] = t + k * T < count ? acc[t + k * T] : l5_one();
        p[k] = k ? mont_call(to_d5(p[k - 1].l), to_d5(a[k].l)) : a[0];
    }
    L5 inv = l5_inverse(p[kInvGroup - 1]);
    _Pragma("unroll") for (int k = kInvGroup - 1; k > 0; k--) {
        const L5x2 x = mont2_call(to_d5(inv.l), to_d5(p[k - 1].l), to_d5(inv.l), to_d5(a[k].l));
        if (t + k * T < count) acc[t + k * T] = x.a;
        inv = x.b;
    }
    if (t < count) acc[t] = inv;
}

template <bool FIRST>
__global__ void __launch_bounds__(kAffThreads, kAffBlocksG1) k_affine_sum_g1(const AffineRound<Fq> a)
{
    const uint32_t np = round_pairs(a), T = gridDim.x * kAffThreads, t0 = blockIdx.x * kAffThreads + threadIdx.x;
    if (t0 >= np) return;
    D5 inv = to_d5(a.acc[t0].l);
    for (uint32_t j = t0 + (np - 1 - t0) / T * T;; j -= T) {
        const uint2 v = pair_at<FIRST>(a, j);
        const D5 pre = unpark(a.out + j);
        Fq x1, x2;
        const bool inf1 = load_x<FIRST>(a.src, v.x, a.nbases, x1), inf2 = load_x<FIRST>(a.src, v.y, a.nbases, x2);
        const Fq y1 = load_y<FIRST>(a.src, v.x, a.nbases), y2 = load_y<FIRST>(a.src, v.y, a.nbases);
        Fq d = sub_plus_p(x2, x1), n = sub_plus_p(y2, y1);
        bool skip = inf1 | inf2, none = inf1 & inf2;
        if (!skip && x1 == x2) {
            const Doubling<Fq> e = same_x(x1, y1, y2);
            d = e.den;
            n = e.num;
            skip = none = !e.ok;
        }
        D5 D = to_d5<0>(d);
        if (skip) D = d5_one();
        const L5x2 w = mont2_call(inv, pre, inv, D);
        inv = to_d5(w.b.l);
        const D5 L = mont_d5(to_d5<0>(n), to_d5(w.a.l));
        Fq x3 = sub(sub(canon52(mont_sqr_call(L).l), x1), x2);
        Fq y3 = sub(mont_fq(L, to_d5<2>(sub_plus_p(x1, x3))), y1);
        if (skip) {
            x3 = none ? marker<Fq>() : inf1 ? x2 : x1;
            y3 = inf1 ? y2 : y1;
        }
        st_elem(&a.out[j].x, x3);
        st_elem(&a.out[j].y, y3);
        if (j < T) break;
    }
}

// limbs of k p - a, k = 2 or 8, for the limbs of a <= k p
template <int K>
__device__ __forceinline__ void neg52(uint64_t n[5], const uint64_t a[5])
{
    constexpr uint64_t p2[5] = {0x1182db0f9fa8eull, 0x22d0e3951a784ull, 0x302b0bb2f02d5ull, 0x405370a08b6d0ull,
                                0x60c89ce5c263ull};
    constexpr uint64_t p8[5] = {0x460b6c3e7ea38ull, 0x8b438e5469e10ull, 0xc0ac2ecbc0b54ull, 0x14dc2822db40ull, 0x183227397098dull};
    int64_t c = 0;
    _Pragma("unroll") for (int i = 0; i < 5; i++) {
        const int64_t x = (int64_t)((K == 2 ? p2[i] : p8[i]) - a[i]) + c;
        n[i] = (uint64_t)x & kM52;
        c = x >> 52;
    }
}
// (a0 b0 + a1 b1) / 2^260 mod p, < 2p for a0 b0 + a1 b1 < p 2^260: two
// products into the same columns, one reduction
static __device__ __noinline__ L5 mont_dot_call(const D5 a0, const D5 b0, const D5 a1, const D5 b1)
{
    L5 r;
    uint64_t c[10];
    _Pragma("unroll") for (int k = 0; k < 10; k++) c[k] = 0 - 2 * prod_bias52(k);
    prod_cols52(c, a0.d, b0.d);
    prod_cols52(c, a1.d, b1.d);
    redc52<FqP>(r.l, c);
    return r;
}

// G2: as G1, with the denominators' norms in the batched inversion,
// 1 / (d0 + d1 i) = (d0 - d1 i) / (d0^2 + d1^2): one norm, 3 Fq products for
// the batch and 2 for the conjugate, against 3 Fq2 products.  The norm is
// parked beside the prefix.  All products are two out-of-line bodies (a
// product, a sum of two products), which keeps the kernels' code small.
template <bool FIRST>
__device__ __forceinline__ L5 pair_norm(const Aff<Fq2>* src, uint64_t nbases, uint2 v, const Fq2& x1, const Fq2& x2, bool skip)
{
    Fq2 d{sub_plus_p(x2.c0, x1.c0), sub_plus_p(x2.c1, x1.c1)};
    if (!skip && x1 == x2) {
        const Doubling<Fq2> e = same_x(x1, load_y<FIRST>(src, v.x, nbases), load_y<FIRST>(src, v.y, nbases));
        d = e.den;
        skip = !e.ok;
    }
    const D5 d0 = to_d5<0>(d.c0), d1 = to_d5<0>(d.c1);
    L5 N = mont_dot_call(d0, d0, d1, d1);
    if (skip) N = l5_one();
    return N;
}

template <bool FIRST>
__global__ void __launch_bounds__(kAffThreads, kAffBlocksG2) k_affine_prefix_g2(const AffineRound<Fq2> a)
{
    const uint32_t np = round_pairs(a), T = gridDim.x * kAffThreads, t0 = blockIdx.x * kAffThreads + threadIdx.x;
    L5 acc = l5_one();
    for (uint32_t j = t0; j < np; j += T) {
        const uint2 v = pair_at<FIRST>(a, j);
        Fq2 x1, x2;
        bool skip = load_x<FIRST>(a.src, v.x, a.nbases, x1);
        skip |= load_x<FIRST>(a.src, v.y, a.nbases, x2);
        char* s = reinterpret_cast<char*>(a.out + j);
        park(s, acc);
        const L5 N = pair_norm<FIRST>(a.src, a.nbases, v, x1, x2, skip);
        park(s + 32, N);
        acc = mont_call(to_d5(acc.l), to_d5(N.l));
    }
    a.acc[t0] = acc;
}

template <bool FIRST>
__global__ void __launch_bounds__(kAffThreads, kAffBlocksG2) k_affine_sum_g2(const AffineRound<Fq2> a)
{
    const uint32_t np = round_pairs(a), T = gridDim.x * kAffThreads, t0 = blockIdx.x * kAffThreads + threadIdx.x;
    if (t0 >= np) return;
    D5 inv = to_d5(a.acc[t0].l);
    for (uint32_t j = t0 + (np - 1 - t0) / T * T;; j -= T) {
        const uint2 v = pair_at<FIRST>(a, j);
        const char* s = reinterpret_cast<const char*>(a.out + j);
        const D5 pre = unpark(s), N = unpark(s + 32);
        Fq2 x1, x2;
        const bool inf1 = load_x<FIRST>(a.src, v.x, a.nbases, x1), inf2 = load_x<FIRST>(a.src, v.y, a.nbases, x2);
        bool skip = inf1 | inf2, none = inf1 & inf2;
        const D5 in = mont_d5(inv, pre);
        inv = mont_d5(inv, N);
        // slope (times 4): (n0 + n1 i)(e0 - e1 i), e = d / norm
        D5 L0, L1;
        {
            const Fq2 y1 = load_y<FIRST>(a.src, v.x, a.nbases), y2 = load_y<FIRST>(a.src, v.y, a.nbases);
            Fq2 d{sub_plus_p(x2.c0, x1.c0), sub_plus_p(x2.c1, x1.c1)};
            Fq2 n{sub_plus_p(y2.c0, y1.c0), sub_plus_p(y2.c1, y1.c1)};
            if (!skip && x1 == x2) {
                const Doubling<Fq2> e = same_x(x1, y1, y2);
                d = e.den;
                n = e.num;
                skip = none = !e.ok;
            }
            const D5 n0 = to_d5<0>(n.c0), n1 = to_d5<0>(n.c1);
            const D5 e0 = mont_d5(to_d5<0>(d.c0), in);
            const L5 e1 = mont_call(to_d5<0>(d.c1), in);
            L5 e1n;
            neg52<2>(e1n.l, e1.l);
            L0 = to_d5(mont_dot_call(n0, e0, n1, to_d5(e1.l)).l);
            L1 = to_d5(mont_dot_call(n1, e0, n0, to_d5(e1n.l)).l);
        }
        Fq2 x3, y3;
        {
            L5 l, ln;
            _Pragma("unroll") for (int i = 0; i < 5; i++) l.l[i] = (uint64_t)__double_as_longlong(__dadd_rn(L1.d[i], 0x1p52)) & kM52;
            neg52<2>(ln.l, l.l);
            x3.c0 = canon52(mont_dot_call(L0, L0, L1, to_d5(ln.l)).l);
            x3.c1 = dbl(mont_fq(L0, L1));
            x3 = sub(sub(x3, x1), x2);
        }
        {
            const D5 w0 = to_d5<2>(sub_plus_p(x1.c0, x3.c0));
            const Fq u = sub_plus_p(x1.c1, x3.c1);
            L5 l, ln;
            to_limbs52<2>(l.l, u.v);
            neg52<8>(ln.l, l.l);
            y3.c0 = canon52(mont_dot_call(L0, w0, L1, to_d5(ln.l)).l);
            y3.c1 = canon52(mont_dot_call(L0, to_d5(l.l), L1, w0).l);
            const Fq2 y1 = load_y<FIRST>(a.src, v.x, a.nbases);
            y3 = sub(y3, y1);
            if (skip) {
                x3 = none ? marker<Fq2>() : inf1 ? x2 : x1;
                y3 = inf1 ? load_y<FIRST>(a.src, v.y, a.nbases) : y1;
            }
        }
        st_elem(&a.out[j].x, x3);
        st_elem(&a.out[j].y, y3);
        if (j < T) break;
    }
}

}  // namespace lzk
