// ntt.cu -- number-theoretic transforms over BN254 Fr.
//
// Replaces number_theory_transformation and its kernels (reference
// include/operator/poly.cuh:32-73): same transform, X_k = sum_j a_j w^(jk)
// in natural order with w the 2^k-th root of unity of ntt-params.cuh
// (w_k = w_28^(2^(28-k)), w_28 = 5^((r-1)/2^28)), and the same radix-2
// decimation-in-frequency butterfly c[j] = lo + hi, c[j^h] = (lo - hi) *
// w^((j mod h) << s).  Instead of one global-memory launch per stage, each
// pass runs m stages on 2^m-element groups, two stages at a time in registers
// and shared memory between them (ceil(k / 10) passes of about equal m for
// blocks of 1024 elements); the scale n^-1 and the coset factors are applied
// as the first pass loads or the last one stores, and a final pass permutes
// in place into natural order.
//
// Directions: forward; inverse (w^-1, then * n^-1); coset forward (a_j *
// g^j first, g = 5 = Fr::multiplicative_generator, alt_bn128_init.cu:50);
// coset inverse (inverse, then * g^-j).
#include "ntt.cuh"
#include "tune.cuh"
#include <map>
#include <mutex>

namespace lzk {

constexpr int kNttMaxLog = 26;
constexpr uint32_t kNttThreads = 256;
constexpr uint32_t kPowLoBits = 12;    // g^j = lo[j & 4095] * hi[j >> 12]

// Montgomery form of w_28 = 5^((r-1)/2^28) and of g = 5
__device__ __forceinline__ Fr root28()
{
    return Fr{{0x80d13d9cu, 0x636e7355u, 0x2445ffd6u, 0xa22bf374u, 0x1eb203d8u, 0x56452ac0u, 0x2963f9e7u, 0x1860ef94u}};
}
__device__ __forceinline__ Fr gen5()
{
    return Fr{{0x9fffffe6u, 0x1b0d0ef9u, 0xa32a913fu, 0xeaba68a3u, 0xd8dd0689u, 0x47d8eb76u, 0x20f5bbc3u, 0x15d00855u}};
}

__device__ __forceinline__ Fr fr_pow(Fr b, uint64_t e)
{
    Fr r = Fr::one();
    while (e) {
        if (e & 1) r = mul(r, b);
        b = sqr(b);
        e >>= 1;
    }
    return r;
}

// consts[0] = w_k, [1] = w_k^-1, [2] = 2^-k, [3] = g, [4] = g^-1,
// [5] = g^(2^12), [6] = g^-(2^12)
__global__ void k_ntt_consts(uint32_t k, Fr* consts)
{
    if (gtid() != 0) return;
    Fr w = root28();
    for (uint32_t i = k; i < 28; i++) w = sqr(w);
    consts[0] = w;
    consts[1] = inverse(w);
    Fr two = add(Fr::one(), Fr::one());
    consts[2] = inverse(fr_pow(two, k));
    Fr g = gen5();
    consts[3] = g;
    consts[4] = inverse(g);
    consts[5] = fr_pow(g, 1ull << kPowLoBits);
    consts[6] = fr_pow(consts[4], 1ull << kPowLoBits);
}

// out[i] = base^i for i < count (64 consecutive powers per thread)
__global__ void k_powers(const Fr* __restrict__ basep, Fr* __restrict__ out, size_t count)
{
    const uint32_t C = 64;
    Fr base = *basep;
    for (uint64_t t = gtid(); t * C < count; t += gstride()) {
        size_t s = t * C;
        Fr v = fr_pow(base, s);
        size_t e = s + C < count ? s + C : count;
        for (size_t i = s; i < e; i++) { st_elem(out + i, v); v = mul(v, base); }
    }
}

// out[i] = in[i] * *scale
__global__ void k_scaled(const Fr* __restrict__ in, const Fr* __restrict__ scale, Fr* __restrict__ out, size_t count)
{
    for (uint64_t i = gtid(); i < count; i += gstride()) st_elem(out + i, mul(ldg_elem(in + i), ldg_elem(scale)));
}

// twiddles in radix-2^52 form: twd[kTwdStride e + i] = limb i of tw[e]
__global__ void k_tw_to_d52(const Fr* __restrict__ tw, double* __restrict__ twd, size_t count)
{
    for (uint64_t e = gtid(); e < count; e += gstride()) {
        double d[5];
        to_d52<0>(d, ldg_elem(tw + e).v);
        double* o = twd + e * kTwdStride;
        _Pragma("unroll") for (int i = 0; i < 5; i++) o[i] = d[i];
        o[5] = 0.0;
    }
}

static std::mutex g_ntt_mu;
static std::map<std::pair<int, uint32_t>, NttTables> g_ntt_tables;
static std::map<int, CosetTables> g_coset_tables;

// Build (once per device and size, synchronously, outside any stream
// capture) the twiddle tables of a size-2^k transform.
int get_tables(uint32_t k, NttTables& out, CosetTables& cos)
{
    int dev;
    LZK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(g_ntt_mu);
    auto it = g_ntt_tables.find({dev, k});
    auto ct = g_coset_tables.find(dev);
    if (it != g_ntt_tables.end() && ct != g_coset_tables.end()) { out = it->second; cos = ct->second; return LZK_OK; }
    cudaStream_t st;
    LZK_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    int rc = LZK_OK;
    const size_t nlo = size_t(1) << kPowLoBits, nhi = size_t(1) << (kNttMaxLog - kPowLoBits);
    if (it == g_ntt_tables.end()) {
        NttTables t;
        size_t half = k ? (size_t(1) << (k - 1)) : 1;
        auto get = [](auto** p, size_t count) { return dev_malloc(reinterpret_cast<void**>(p), count * sizeof(**p)) == LZK_OK; };
        bool ok = get(&t.consts, 8) && get(&t.tw[0], half) && get(&t.tw[1], half) &&
                  get(&t.twd[0], half * kTwdStride) && get(&t.twd[1], half * kTwdStride) && get(&t.slo[0], nlo) &&
                  get(&t.slo[1], nlo);
        CosetTables c;
        const bool coset = ct == g_coset_tables.end();
        if (!coset) c = ct->second;
        for (int d = 0; d < 2 && coset; d++) ok = ok && get(&c.lo[d], nlo) && get(&c.hi[d], nhi);
        if (ok) {
            k_ntt_consts<<<1, 32, 0, st>>>(k, t.consts); note_launch();
            for (int d = 0; d < 2; d++) {
                k_powers<<<grid_for((half + 63) / 64, 128), 128, 0, st>>>(t.consts + d, t.tw[d], half); note_launch();
                k_tw_to_d52<<<grid_for(half, 128), 128, 0, st>>>(t.tw[d], t.twd[d], half); note_launch();
                if (coset) {
                    k_powers<<<grid_for(nlo / 64, 128), 128, 0, st>>>(t.consts + 3 + d, c.lo[d], nlo); note_launch();
                    k_powers<<<grid_for(nhi / 64, 128), 128, 0, st>>>(t.consts + 5 + d, c.hi[d], nhi); note_launch();
                }
                k_scaled<<<grid_for(nlo, 128), 128, 0, st>>>(c.lo[d], t.consts + 2, t.slo[d], nlo); note_launch();
            }
            rc = cuda_status(cudaStreamSynchronize(st));
        } else {
            rc = LZK_ENOMEM;
        }
        if (rc == LZK_OK) {
            g_ntt_tables[{dev, k}] = t;
            g_coset_tables[dev] = c;
        } else {
            void* mine[] = {t.consts, t.tw[0], t.tw[1], t.twd[0], t.twd[1], t.slo[0], t.slo[1]};
            for (auto m : mine) cudaFree(m);
            for (int d = 0; d < 2 && coset; d++) { cudaFree(c.lo[d]); cudaFree(c.hi[d]); }
        }
    }
    cudaStreamDestroy(st);
    if (rc != LZK_OK) return rc;
    out = g_ntt_tables[{dev, k}];
    cos = g_coset_tables[dev];
    return LZK_OK;
}

struct NttPass {
    uint32_t k, s0, m, lowbits, R;
    uint32_t canon;     // the last pass: canonical results
    uint32_t natural;   // a DIF transform of one pass (one block), written in natural order
};

__device__ __forceinline__ size_t brev_k(size_t j, uint32_t k)
{
    return k ? (size_t)(__brevll((unsigned long long)j) >> (64 - k)) : 0;
}

// ---------------- lazily reduced values ----------------
// Inside a pass a value stays below 2p (DIF) or 4p (DIT) instead of p, so a
// butterfly needs one conditional subtraction instead of three.  The FP64
// product of x and t is 16 x t / 2^260 + (less than p), with 2^260 = 84.6 p:
// below 2p for x < 4p and t < 1.3 p (16 4 1.3 = 83.2).  t is a canonical table
// value, or a product of canonical ones (edge_apply2).
__host__ __device__ constexpr uint32_t fr_2p(int i) { return (FrP::p(i) << 1) | (i ? FrP::p(i - 1) >> 31 : 0u); }

// a + b, no reduction
__device__ __forceinline__ Fr add_raw(const Fr& a, const Fr& b)
{
    Fr r;
    add_nored(r.v, a.v, b.v);
    return r;
}
// x < 4p to x mod 2p
__device__ __forceinline__ Fr red_2p(const Fr& x)
{
    uint32_t s[8], br;
    asm("sub.cc.u32  %0, %9,  %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(br)
        : "r"(x.v[0]), "r"(x.v[1]), "r"(x.v[2]), "r"(x.v[3]), "r"(x.v[4]), "r"(x.v[5]), "r"(x.v[6]), "r"(x.v[7]),
          "n"(fr_2p(0)), "n"(fr_2p(1)), "n"(fr_2p(2)), "n"(fr_2p(3)), "n"(fr_2p(4)), "n"(fr_2p(5)), "n"(fr_2p(6)), "n"(fr_2p(7)));
    Fr r;
    _Pragma("unroll") for (int i = 0; i < 8; i++) r.v[i] = br ? x.v[i] : s[i];
    return r;
}
// a + 2p - b for a, b < 2p: in (0, 4p)
__device__ __forceinline__ Fr sub_2p(const Fr& a, const Fr& b)
{
    uint32_t t[8];
    asm("add.cc.u32  %0, %8,  %16;\n\t"
        "addc.cc.u32 %1, %9,  %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "n"(fr_2p(0)), "n"(fr_2p(1)), "n"(fr_2p(2)), "n"(fr_2p(3)), "n"(fr_2p(4)), "n"(fr_2p(5)), "n"(fr_2p(6)), "n"(fr_2p(7)));
    Fr r;
    asm("sub.cc.u32  %0, %8,  %16;\n\t"
        "subc.cc.u32 %1, %9,  %17;\n\t"
        "subc.cc.u32 %2, %10, %18;\n\t"
        "subc.cc.u32 %3, %11, %19;\n\t"
        "subc.cc.u32 %4, %12, %20;\n\t"
        "subc.cc.u32 %5, %13, %21;\n\t"
        "subc.cc.u32 %6, %14, %22;\n\t"
        "subc.u32    %7, %15, %23;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
        : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    return r;
}

// A product operand in radix-2^52 form, and x tx, y ty (< 2p) for x, y < 4p and
// tx, ty < 1.3 p.
// Two products to a call: they interleave, and one body of about 700
// instructions keeps the pass inside the instruction cache.
struct Tw {
    double d[5];
};
struct FrPair {
    Fr a, b;
};
static __device__ __noinline__ FrPair fr_mul2(const Fr x, const Fr y, const Tw tx, const Tw ty)
{
    double dx[5], dy[5];
    uint64_t rx[5], ry[5];
    to_d52<4>(dx, x.v);
    to_d52<4>(dy, y.v);
    mont52_core<FrP>(rx, dx, tx.d);
    mont52_core<FrP>(ry, dy, ty.d);
    FrPair r;
    from_limbs52(r.a.v, rx);
    from_limbs52(r.b.v, ry);
    return r;
}
__device__ __forceinline__ Tw tw_of(const Fr& x)
{
    Tw t;
    to_d52<0>(t.d, x.v);
    return t;
}
// Twiddle e: from the radix-2^52 table (TWD), or converted
template <bool TWD>
__device__ __forceinline__ Tw load_tw(const Fr* __restrict__ tw, const double* __restrict__ twd, uint32_t e)
{
    if (TWD) {
        const double2* q = reinterpret_cast<const double2*>(twd + (size_t)e * kTwdStride);
        const double2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
        return Tw{{a.x, a.y, b.x, b.y, c.x}};
    }
    return tw_of(ldg_elem(tw + e));
}

// Factor a pass applies to each element as it loads it (the first pass) or
// stores it (the last pass): x * scale * g^e, e = the position j, or, with
// brev set, the coefficient index brev(j) that a bit-reversed position
// holds; a null scale or null power tables stand for 1.  x < 4p, result < 2p:
// the table values are canonical, so lo hi < (1 + 16 / 84.6) p = 1.19 p, and
// that times the scale < (1 + 16 1.19 / 84.6) p = 1.23 p.
__device__ __forceinline__ void edge_apply2(const NttEdge& ed, Fr& x, Fr& y, uint32_t jx, uint32_t jy, uint32_t k)
{
    if (ed.lo) {
        if (ed.brev) { jx = (uint32_t)brev_k(jx, k); jy = (uint32_t)brev_k(jy, k); }
        const uint32_t m = (1u << kPowLoBits) - 1;
        FrPair c = fr_mul2(ldg_elem(ed.lo + (jx & m)), ldg_elem(ed.lo + (jy & m)), tw_of(ldg_elem(ed.hi + (jx >> kPowLoBits))),
                           tw_of(ldg_elem(ed.hi + (jy >> kPowLoBits))));
        if (ed.scale) {
            const Tw s = tw_of(ldg_elem(ed.scale));
            c = fr_mul2(c.a, c.b, s, s);
        }
        c = fr_mul2(x, y, tw_of(c.a), tw_of(c.b));
        x = c.a; y = c.b;
    } else if (ed.scale) {
        const Tw s = tw_of(ldg_elem(ed.scale));
        const FrPair c = fr_mul2(x, y, s, s);
        x = c.a; y = c.b;
    }
}

// m radix-2 stages over groups of 2^m elements that differ in index bits
// [lowbits, lowbits+m); R groups with consecutive (outer, low) index per
// block.  `batch` transforms of size 2^k lie `bstride` elements apart (or at
// ptrs[blockIdx.y]).
//   DIF (decimation in frequency): stages s0 .. s0+m-1, natural order in,
//     bit-reversed out after all passes; c[j] = lo + hi, c[j^h] =
//     (lo - hi) w^((j mod h) << s) (poly.cuh:38-39).
//   DIT (decimation in time): stages t = lowbits .. lowbits+m-1, bit-reversed
//     order in, natural out; with u = w^((j mod 2^t) << (k-1-t)) hi,
//     c[j] = lo + u, c[j + 2^t] = lo - u.
// Both compute X_k = sum_j a_j w^(jk).
//
// A thread takes four elements a quarter of a radix-4 span apart and runs two
// stages on them in registers (one stage first when m is odd); shared memory
// holds the block between the steps, the first step reads and the last writes
// global memory.  Shared memory is two planes of 16-byte halves, swizzled so
// that the strided reads of the short spans spread over the banks.
//
// Bound by the issue of the products (325 instructions of about 460 a
// butterfly).  Against one stage at a time on canonical values, bit reversal
// included: 2^12 forward 41.0 -> 32.8 us, 2^20 coset forward 323 -> 296, 2^24
// coset inverse 6713 -> 5102.  Three blocks a multiprocessor instead of two
// (80 registers) spilled and was 12 % slower.
__device__ __forceinline__ uint32_t swz(uint32_t i) { return i ^ ((i >> 2) & 7u); }

template <bool DIT, bool TWD>
__global__ void __launch_bounds__(kNttThreads, 2) k_ntt_pass(Fr* __restrict__ data, NttPass p, const Fr* __restrict__ tw,
                                                             const double* __restrict__ twd, NttEdge pre, NttEdge post,
                                                             size_t bstride, Fr* const* __restrict__ ptrs)
{
    extern __shared__ uint4 sm[];
    Fr* d = ptrs ? ptrs[blockIdx.y] : data + (size_t)blockIdx.y * bstride;
    const uint32_t rbits = __ffs(p.R) - 1, tot = p.R << p.m, units = tot >> 2;
    const uint32_t lowmask = (1u << p.lowbits) - 1;
    auto sm_ld = [&](uint32_t i) -> Fr {
        Fr x;
        uint4* q = reinterpret_cast<uint4*>(&x);
        q[0] = sm[swz(i)];
        q[1] = sm[tot + swz(i)];
        return x;
    };
    auto sm_st = [&](uint32_t i, const Fr& x) {
        const uint4* q = reinterpret_cast<const uint4*>(&x);
        sm[swz(i)] = q[0];
        sm[tot + swz(i)] = q[1];
    };
    // steps of two stages: quarter spans 2^h; an odd count starts with one stage
    const uint32_t steps = (p.m + 1) >> 1;
    for (uint32_t st = 0; st < steps; st++) {
        const bool first = st == 0, last = st + 1 == steps, odd = (p.m & 1) != 0, one = first && odd;
        // stages done before this step: 2 st, or 2 st - 1 after an odd start
        const uint32_t done = 2 * st - (odd && st ? 1u : 0u);
        const uint32_t h = DIT ? done : one ? p.m - 2 : p.m - 2 - done;
        for (uint32_t u = threadIdx.x; u < units; u += blockDim.x) {
            const uint32_t r = u & (p.R - 1), gq = u >> rbits, gl = gq & ((1u << h) - 1);
            const uint32_t g0 = ((gq >> h) << (h + 2)) | gl;
            const uint32_t cidx = blockIdx.x * p.R + r, low = cidx & lowmask;
            const uint32_t j0 = ((cidx >> p.lowbits) << (p.lowbits + p.m)) | (g0 << p.lowbits) | low, js = 1u << (h + p.lowbits);
            const uint32_t i0 = (g0 << rbits) | r, is = 1u << (h + rbits);
            const uint32_t jm = (gl << p.lowbits) | low;
            // twiddle exponent shift of the stage whose two pairs share one
            // twiddle (1 in the transform's first DIT or last DIF stage);
            // loading a step's twiddles ahead of its elements spilled: 13 %
            // slower
            const uint32_t e = DIT ? p.k - 1 - (p.lowbits + h) : p.s0 + p.m - 1 - h;
            const bool unit = p.lowbits + h == 0;
            Fr x0, x1, x2, x3;
            if (first) {
                x0 = ld_elem(d + j0);
                x1 = ld_elem(d + j0 + js);
                x2 = ld_elem(d + j0 + 2 * js);
                x3 = ld_elem(d + j0 + 3 * js);
                if (pre.lo || pre.scale) {
                    edge_apply2(pre, x0, x1, j0, j0 + js, p.k);
                    edge_apply2(pre, x2, x3, j0 + 2 * js, j0 + 3 * js, p.k);
                }
            } else {
                x0 = sm_ld(i0);
                x1 = sm_ld(i0 + is);
                x2 = sm_ld(i0 + 2 * is);
                x3 = sm_ld(i0 + 3 * is);
            }
            if (DIT) {
                // stage h on (x0, x1), (x2, x3)
                if (unit) {
                    x1 = red_2p(x1);
                    x3 = red_2p(x3);
                } else {
                    const Tw t = load_tw<TWD>(tw, twd, jm << e);
                    const FrPair v = fr_mul2(x1, x3, t, t);
                    x1 = v.a; x3 = v.b;
                }
                x0 = red_2p(x0);
                x2 = red_2p(x2);
                Fr t0 = add_raw(x0, x1), t2 = add_raw(x2, x3);
                x1 = sub_2p(x0, x1);
                x3 = sub_2p(x2, x3);
                x0 = t0;
                x2 = t2;
                if (!one) {
                    // stage h + 1 on (x0, x2), (x1, x3)
                    const FrPair v = fr_mul2(x2, x3, load_tw<TWD>(tw, twd, jm << (e - 1)),
                                             load_tw<TWD>(tw, twd, (jm + js) << (e - 1)));
                    x0 = red_2p(x0);
                    x1 = red_2p(x1);
                    x2 = sub_2p(x0, v.a);
                    x3 = sub_2p(x1, v.b);
                    x0 = add_raw(x0, v.a);
                    x1 = add_raw(x1, v.b);
                }
            } else {
                // stage h + 1 on (x0, x2), (x1, x3)
                Fr t0 = red_2p(add_raw(x0, x2)), t1 = red_2p(add_raw(x1, x3));
                const FrPair v = fr_mul2(sub_2p(x0, x2), sub_2p(x1, x3), load_tw<TWD>(tw, twd, jm << (e - 1)),
                                         load_tw<TWD>(tw, twd, (jm + js) << (e - 1)));
                x0 = t0; x1 = t1; x2 = v.a; x3 = v.b;
                if (!one) {
                    // stage h on (x0, x1), (x2, x3)
                    t0 = red_2p(add_raw(x0, x1));
                    t1 = red_2p(add_raw(x2, x3));
                    x1 = sub_2p(x0, x1);
                    x3 = sub_2p(x2, x3);
                    if (unit) {
                        x1 = red_2p(x1);
                        x3 = red_2p(x3);
                    } else {
                        const Tw t = load_tw<TWD>(tw, twd, jm << e);
                        const FrPair z = fr_mul2(x1, x3, t, t);
                        x1 = z.a; x3 = z.b;
                    }
                    x0 = t0;
                    x2 = t1;
                }
            }
            if (last) {
                if (post.lo || post.scale) {
                    edge_apply2(post, x0, x1, j0, j0 + js, p.k);
                    edge_apply2(post, x2, x3, j0 + 2 * js, j0 + 3 * js, p.k);
                } else if (DIT && p.canon) {
                    x0 = red_2p(x0); x1 = red_2p(x1); x2 = red_2p(x2); x3 = red_2p(x3);
                }
                if (p.canon) {
                    x0 = final_sub<FrP>(x0.v); x1 = final_sub<FrP>(x1.v);
                    x2 = final_sub<FrP>(x2.v); x3 = final_sub<FrP>(x3.v);
                }
                auto at = [&](uint32_t j) { return p.natural ? (uint32_t)brev_k(j, p.k) : j; };
                st_elem(d + at(j0), x0);
                st_elem(d + at(j0 + js), x1);
                st_elem(d + at(j0 + 2 * js), x2);
                st_elem(d + at(j0 + 3 * js), x3);
            } else {
                sm_st(i0, x0);
                sm_st(i0 + is, x1);
                sm_st(i0 + 2 * is, x2);
                sm_st(i0 + 3 * is, x3);
            }
        }
        if (!last) __syncthreads();
    }
}

// The transform of two elements (k = 1), both factors and directions alike:
// x0 + x1, x0 - x1 with the edges of the one pass.
__global__ void k_ntt_two(Fr* __restrict__ data, NttEdge pre, NttEdge post, size_t bstride, Fr* const* __restrict__ ptrs)
{
    if (threadIdx.x) return;
    Fr* d = ptrs ? ptrs[blockIdx.x] : data + (size_t)blockIdx.x * bstride;
    Fr x = ld_elem(d), y = ld_elem(d + 1);
    edge_apply2(pre, x, y, 0, 1, 1);
    x = final_sub<FrP>(x.v);
    y = final_sub<FrP>(y.v);
    Fr a = add(x, y), b = sub(x, y);
    edge_apply2(post, a, b, 0, 1, 1);
    st_elem(d, final_sub<FrP>(a.v));
    st_elem(d + 1, final_sub<FrP>(b.v));
}

// A transform of 2^k elements, 2 <= k <= kNttShortLog, in one block: a
// butterfly a thread and stage, natural order out.  The chain of stages bounds
// it; a pass of k_ntt_pass, two stages on four elements a thread, has pairs of
// products, and the factors of four elements one after the other, in that
// chain.  Coset forward at 2^6 and 2^8, 200 calls in a row: 8.2 and 10.3 us a
// call (8 is the launch), with a pass 16.4 and 19.5, a stage at a time on
// canonical values with a reversal 11.5 and 16.4.  At 2^9 one transform takes
// 15.4 instead of 22.6 us, but 16384 of them 788 instead of 744: there the
// passes stay.
constexpr uint32_t kNttShortLog = 8;
template <bool TWD>
__global__ void __launch_bounds__(1 << (kNttShortLog - 1)) k_ntt_short(Fr* __restrict__ data, uint32_t k, const Fr* __restrict__ tw,
                                                                       const double* __restrict__ twd, NttEdge pre, NttEdge post,
                                                                       size_t bstride, Fr* const* __restrict__ ptrs)
{
    __shared__ uint4 sm[2 << kNttShortLog];
    Fr* d = ptrs ? ptrs[blockIdx.x] : data + (size_t)blockIdx.x * bstride;
    const uint32_t t = threadIdx.x, n = 1u << k;
    uint32_t j = t, h = n >> 1;
    Fr x = ld_elem(d + j), y = ld_elem(d + j + h);
    edge_apply2(pre, x, y, j, j + h, k);
    for (uint32_t s = 0;; s++) {
        const Fr b = sub_2p(x, y);
        x = red_2p(add_raw(x, y));
        if (h == 1) {   // the last stage's twiddles are 1
            y = red_2p(b);
            break;
        }
        const Tw w = load_tw<TWD>(tw, twd, (t & (h - 1)) << s);
        double db[5];
        uint64_t r[5];
        to_d52<4>(db, b.v);
        mont52_core<FrP>(r, db, w.d);
        from_limbs52(y.v, r);
        const uint4 *xq = reinterpret_cast<const uint4*>(&x), *yq = reinterpret_cast<const uint4*>(&y);
        sm[j] = xq[0]; sm[n + j] = xq[1];
        sm[j + h] = yq[0]; sm[n + j + h] = yq[1];
        __syncthreads();
        h >>= 1;
        j = 2 * t - (t & (h - 1));
        uint4 *xo = reinterpret_cast<uint4*>(&x), *yo = reinterpret_cast<uint4*>(&y);
        xo[0] = sm[j]; xo[1] = sm[n + j];
        yo[0] = sm[j + h]; yo[1] = sm[n + j + h];
    }
    edge_apply2(post, x, y, j, j + h, k);
    st_elem(d + brev_k(j, k), final_sub<FrP>(x.v));
    st_elem(d + brev_k(j + h, k), final_sub<FrP>(y.v));
}

// In-place bit reversal, element by element (short transforms).
__global__ void k_ntt_bitrev(Fr* __restrict__ data, uint32_t k, size_t bstride, Fr* const* __restrict__ ptrs)
{
    Fr* d = ptrs ? ptrs[blockIdx.y] : data + (size_t)blockIdx.y * bstride;
    const size_t n = size_t(1) << k;
    for (uint64_t j = gtid(); j < n; j += gstride()) {
        const size_t r = brev_k(j, k);
        if (j >= r) continue;
        const Fr a = ld_elem(d + j), b = ld_elem(d + r);
        st_elem(d + r, a);
        st_elem(d + j, b);
    }
}

// In-place bit reversal by tiles.  With the index split into (H, M, L), H and
// L of 5 bits, (H, M, L) goes to (brev L, brev M, brev H): the 32 x 32 tile of
// M, rows of 1 KB, is the tile of brev M transposed with its rows and columns
// bit-reversed.  A block exchanges tiles M and brev M through shared memory,
// so every access to global memory is a full row; element by element the
// writes touch one 32-byte sector at a time.  (In a 2^24 coset inverse the
// element-wise form took 2080 us, factors included; those are now applied by
// the last pass.)  A row enters shared memory at its bit-reversed number, so that a column is
// read at the odd stride of 33 units.
constexpr uint32_t kTileRow = 33, kTile = 32 * kTileRow;
__global__ void __launch_bounds__(256) k_ntt_bitrev_tiles(Fr* __restrict__ data, uint32_t k, size_t bstride,
                                                          Fr* const* __restrict__ ptrs)
{
    extern __shared__ uint4 sm[];   // two tiles, two planes each
    const uint32_t mb = k - 10, M = blockIdx.x, N = mb ? __brev(M) >> (32 - mb) : 0;
    if (M > N) return;
    Fr* d = ptrs ? ptrs[blockIdx.y] : data + (size_t)blockIdx.y * bstride;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, tiles = M == N ? 1 : 2;
    for (uint32_t t = 0; t < tiles; t++) {
        const Fr* src = d + ((size_t)(t ? N : M) << 5) + lane;
        uint4* q = sm + t * 2 * kTile + lane;
        for (uint32_t row = w; row < 32; row += 8) {
            const Fr x = ld_elem(src + ((size_t)row << (k - 5)));
            const uint32_t at = (__brev(row) >> 27) * kTileRow;
            q[at] = reinterpret_cast<const uint4*>(&x)[0];
            q[kTile + at] = reinterpret_cast<const uint4*>(&x)[1];
        }
    }
    __syncthreads();
    for (uint32_t t = 0; t < tiles; t++) {
        // tile t of the source fills the other tile
        Fr* dst = d + ((size_t)(t ? M : N) << 5) + lane;
        const uint4* q = sm + t * 2 * kTile + lane * kTileRow;
        for (uint32_t row = w; row < 32; row += 8) {
            Fr x;
            const uint32_t at = __brev(row) >> 27;
            reinterpret_cast<uint4*>(&x)[0] = q[at];
            reinterpret_cast<uint4*>(&x)[1] = q[kTile + at];
            st_elem(dst + ((size_t)row << (k - 5)), x);
        }
    }
}

// the one element of a transform of size 1 times its scale
__global__ void k_ntt_one(Fr* __restrict__ data, const Fr* __restrict__ scale, size_t bstride, Fr* const* __restrict__ ptrs)
{
    if (threadIdx.x) return;
    Fr* d = ptrs ? ptrs[blockIdx.x] : data + (size_t)blockIdx.x * bstride;
    st_elem(d, mul(ld_elem(d), ldg_elem(scale)));
}

int ntt_prepare_launch()
{
    static std::mutex mu;
    static bool attr_set[64] = {false};
    int dev = 0;
    LZK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        // the largest block the tuning table allows (kMaxNttBlock elements)
        LZK_CUDA(cudaFuncSetAttribute(k_ntt_pass<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxNttBlock * sizeof(Fr)));
        LZK_CUDA(cudaFuncSetAttribute(k_ntt_pass<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxNttBlock * sizeof(Fr)));
        LZK_CUDA(cudaFuncSetAttribute(k_ntt_pass<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxNttBlock * sizeof(Fr)));
        LZK_CUDA(cudaFuncSetAttribute(k_ntt_pass<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxNttBlock * sizeof(Fr)));
        LZK_CUDA(cudaFuncSetAttribute(k_ntt_bitrev_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kTile * sizeof(uint4)));
        attr_set[dev] = true;
    }
    return LZK_OK;
}

// Whether a transform of size 2^k is one pass of several steps, whose only
// block has read every element when it writes the first one: such a DIF
// transform writes its results in natural order itself.
static bool ntt_one_pass(uint32_t k, uint32_t block) { return k > 2 && k < 32 && (1u << k) <= block; }

int ntt_passes(Fr* data, uint32_t k, uint32_t count, size_t bstride, const Fr* tw, bool dit, NttEdge pre,
               NttEdge post, cudaStream_t st, Fr* const* ptrs, const double* twd, uint32_t elems, bool natural)
{
    if (k == 0 || k > 30 || count == 0 || count > 65535 || (!data && !ptrs) || !tw) return LZK_EINVAL;
    LZK_TRY(ntt_prepare_launch());
    if (k == 1) {
        k_ntt_two<<<count, 32, 0, st>>>(data, pre, post, bstride, ptrs); note_launch();
        return launch_status();
    }
    // blocks of 2^maxm elements, at most maxm stages a pass
    if (!elems) elems = tune_ntt_block(k);
    uint32_t maxm = 0;
    while ((1u << (maxm + 1)) <= elems) maxm++;
    const uint32_t P = (k + maxm - 1) / maxm;
    const size_t n = size_t(1) << k;
    uint32_t done = 0;   // stages done by earlier passes
    for (uint32_t q = 0; q < P; q++) {
        uint32_t m = (k - done) / (P - q);    // balanced split, larger passes last
        NttPass pp;
        pp.k = k; pp.m = m;
        // DIF passes take the top index bits first, DIT passes the bottom ones
        pp.lowbits = dit ? done : k - done - m;
        pp.s0 = dit ? 0 : done;
        uint32_t G = 1u << m;
        uint32_t R = elems / G;
        if ((size_t)R > (n >> m)) R = (uint32_t)(n >> m);
        if (R == 0) R = 1;
        pp.R = R;
        pp.canon = q == P - 1;
        pp.natural = natural;
        const unsigned threads = G * R / 4 < kNttThreads ? G * R / 4 : kNttThreads;
        size_t blocks = (n >> m) / R;
        size_t smem = (size_t)G * R * sizeof(Fr);
        NttEdge a = q == 0 ? pre : NttEdge{}, b = q == P - 1 ? post : NttEdge{};
        const dim3 grid((unsigned)blocks, count);
        if (dit && twd)
            k_ntt_pass<true, true><<<grid, threads, smem, st>>>(data, pp, tw, twd, a, b, bstride, ptrs);
        else if (dit)
            k_ntt_pass<true, false><<<grid, threads, smem, st>>>(data, pp, tw, twd, a, b, bstride, ptrs);
        else if (twd)
            k_ntt_pass<false, true><<<grid, threads, smem, st>>>(data, pp, tw, twd, a, b, bstride, ptrs);
        else
            k_ntt_pass<false, false><<<grid, threads, smem, st>>>(data, pp, tw, twd, a, b, bstride, ptrs);
        note_launch();
        done += m;
    }
    return launch_status();
}

// Enqueue `count` transforms of size 2^k (natural order in, natural order
// out) with twiddle table tw (w^e, e < n/2): DIF passes with the input and
// output factors, then the bit reversal.
static int ntt_enqueue(Fr* data, uint32_t k, uint32_t count, size_t bstride, const Fr* tw, NttEdge pre, NttEdge post,
                       cudaStream_t st, Fr* const* ptrs = nullptr, const double* twd = nullptr)
{
    LZK_TRY(ntt_prepare_launch());
    if (k == 0) {
        // g^0 = 1: only a scale is left
        if (!post.scale) return LZK_OK;
        k_ntt_one<<<count, 32, 0, st>>>(data, post.scale, bstride, ptrs); note_launch();
        return launch_status();
    }
    if (k > 1 && k <= kNttShortLog) {
        if (twd) k_ntt_short<true><<<count, 1u << (k - 1), 0, st>>>(data, k, tw, twd, pre, post, bstride, ptrs);
        else k_ntt_short<false><<<count, 1u << (k - 1), 0, st>>>(data, k, tw, twd, pre, post, bstride, ptrs);
        note_launch();
        return launch_status();
    }
    // one look at the tuning table, which another thread may be setting: the
    // passes and the reversal have to agree on it
    const uint32_t block = tune_ntt_block(k);
    const bool one = ntt_one_pass(k, block);
    LZK_TRY(ntt_passes(data, k, count, bstride, tw, false, pre, post, st, ptrs, twd, block, one));
    if (k < 2 || one) return launch_status();
    if (k < 10) {
        k_ntt_bitrev<<<dim3(grid_for(size_t(1) << k, 256), count), 256, 0, st>>>(data, k, bstride, ptrs); note_launch();
    } else {
        k_ntt_bitrev_tiles<<<dim3(1u << (k - 10), count), 256, 4 * kTile * sizeof(uint4), st>>>(data, k, bstride, ptrs); note_launch();
    }
    return launch_status();
}

int ntt_run(Fr* data, uint32_t k, int dir, uint32_t count, size_t bstride, const Fr* scale_override, cudaStream_t st,
            Fr* const* ptrs)
{
    if ((!data && !ptrs) || k > kNttMaxLog || dir < 0 || dir > 3 || count == 0 || count > 65535) return LZK_EINVAL;
    if (!ptrs && count > 1 && bstride < (size_t(1) << k)) return LZK_EINVAL;
    NttTables t; CosetTables c;
    LZK_TRY(get_tables(k, t, c));
    bool inv = dir & 1, coset = dir >= 2;
    NttEdge pre, post;
    if (coset && !inv) pre = NttEdge{c.lo[0], c.hi[0], nullptr, 0};
    if (coset && inv) {
        // h_j = (...) n^-1 g^-j of the coefficient j that position brev(j) holds
        post = scale_override ? NttEdge{c.lo[1], c.hi[1], scale_override, 1} : NttEdge{t.slo[1], c.hi[1], nullptr, 1};
    } else {
        post.scale = scale_override ? scale_override : inv ? t.consts + 2 : nullptr;
    }
    return ntt_enqueue(data, k, count, bstride, t.tw[inv ? 1 : 0], pre, post, st, ptrs, twd_for(t, inv ? 1 : 0, k));
}

}  // namespace lzk

using namespace lzk;

extern "C" {

int lzk_ntt_prepare(uint32_t log_n)
{
    if (log_n > kNttMaxLog) return LZK_EINVAL;
    NttTables t; CosetTables c;
    return get_tables(log_n, t, c);
}

int lzk_ntt(lzk_fr_t* data, uint32_t log_n, int direction, void* stream)
{
    return ntt_run(reinterpret_cast<Fr*>(data), log_n, direction, 1, 0, nullptr, as_stream(stream));
}

int lzk_ntt_batch(lzk_fr_t* data, uint32_t log_n, uint32_t count, size_t stride, int direction, void* stream)
{
    return ntt_run(reinterpret_cast<Fr*>(data), log_n, direction, count, stride, nullptr, as_stream(stream));
}

int lzk_number_theory_transformation(size_t deg, size_t log_deg, lzk_fr_t* coeffs, const lzk_fr_t* omega_powers,
                                     const lzk_fr_t* factor, void* stream)
{
    if (!coeffs || !omega_powers || log_deg > 30 || deg != (size_t(1) << log_deg)) return LZK_EINVAL;
    return ntt_enqueue(reinterpret_cast<Fr*>(coeffs), (uint32_t)log_deg, 1, 0,
                       reinterpret_cast<const Fr*>(omega_powers), NttEdge{},
                       NttEdge{nullptr, nullptr, reinterpret_cast<const Fr*>(factor), 0}, as_stream(stream));
}

}  // extern "C"
