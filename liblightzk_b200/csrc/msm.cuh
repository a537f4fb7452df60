// msm.cuh -- shared pieces of the Pippenger MSM (msm_sort.cu, msm_g1.cu,
// msm_g2.cu).  See msm_sort.cu for the pipeline.
#pragma once
#include "common.cuh"
#include "curve.cuh"
#include "glv.cuh"
#include "tune.cuh"

namespace lzk {

// G2 points over two lanes (curve.cuh)
template <class F> struct LaneOf { using T = F; };
template <> struct LaneOf<Fq2> { using T = Fq2P; };

struct G1 { using F = Fq; };
struct G2 { using F = Fq2; };

constexpr uint32_t kLevelL = 32;     // smallest warp tile of the bucket reduction (scratch bound)
constexpr uint32_t kFixSmall = 64;   // partials a single fix-up thread folds

// Batched affine rounds before the XYZZ accumulation (affine.cuh).
constexpr uint32_t kNoEntry = 0xffffffffu;   // a gap in the padded entry list
constexpr int kLayoutPoints = 16;            // accumulation operands: the points the rounds leave
constexpr uint32_t kAffMaxRounds = 5;
// threads a block and blocks an SM holds (128 and 254 registers; 3 or 5
// blocks for G1, 3 or 4 for G2 measured slower)
constexpr uint32_t kAffThreads = 128, kAffBlocksG1 = 4, kAffBlocksG2 = 2;
constexpr unsigned kAffMinPairs = 4;   // pairs a thread takes at least
constexpr int kInvGroup = 4;           // products an inverting thread takes
// Slots whose rounds run together, a bound on the scratch (48 bytes a slot for
// G1, 96 for G2).  Each slice pays its rounds' inversions (29 us) again: the
// proof at 2^20 takes 21.0 ms with 2^24, 22.2 with 2^23 (G1) and 2^22 (G2).
constexpr size_t kAffSlice = size_t(1) << 24;
// Rounds R for `entries` sorted entries over B buckets: as long as a bucket
// still holds fill 2^R entries on average.  Gaps that pad buckets to multiples
// of 2^R then stay below a tenth (fill 8, one bucket set for all windows) or a
// fifth of the slots (fill 4, a set per window: buckets are shorter there, and
// a G2 MSM of 250000 plain points takes 4919 instead of 5529 us; a G1 table
// MSM of 66000 points 632 instead of 595).  At 2^20 over a table (240 entries
// a bucket) R = 1 .. 4 measured 3480, 3279, 3204, 3207 us, against 3641 us
// without rounds.  Lists shorter than kAffMinEntries run at the latency of the
// rounds' launches.
constexpr size_t kAffMinEntries = 1u << 16, kAffFillTable = 8, kAffFillPlain = 4;
inline uint32_t affine_rounds(size_t entries, size_t B, size_t fill)
{
    uint32_t R = 0;
    if (entries < kAffMinEntries) return 0;
    while (R < kAffMaxRounds && entries >= (B << (R + 1)) * fill) R++;
    // slot numbers are 32 bits
    return entries + (B << R) < (1ull << 32) ? R : 0;
}

struct MsmPlan {
    size_t n = 0;
    uint32_t c = 0;        // window bits
    uint32_t W = 0;        // digit windows
    uint32_t nb = 0;       // buckets per window = 2^(c-1)
    uint32_t wb = 0;       // bucket sets: W (plain) or 1 (shared, precomputed)
    uint32_t B = 0;        // total buckets = wb * nb
    bool shared = false;   // precomputed table: one bucket set for all windows
    size_t stride = 0;     // table level stride
    size_t max_entries = 0;
    uint32_t chunk = 0;    // sorted entries per accumulation thread
    uint32_t run = 0;      // buckets per lane run of the reduction tiles
    size_t chunks = 0;
    bool glv = false;         // plain G1: every scalar in two halves, over 2 n bases (glv.cuh)
    uint32_t rounds = 0;      // batched affine rounds before the accumulation
    size_t max_slots = 0;     // entries with the gaps that pad buckets to 2^rounds
    size_t slice = 0;         // slots a slice
    // workspace offsets
    size_t o_cnt, o_off, o_ent, o_bsum, o_head, o_tail, o_lr0, o_la0, o_lr1, o_la1, o_scan, o_large, o_aff, o_fin, o_phi,
        bytes;
};

// One affine round (affine.cuh) of slots [s0, s0 + slots) of a padded entry
// list of *total slots: src are the bases (r = 1) or the slice's points of the
// round before, out its results, r the rounds done after this one, acc a
// product per thread.
struct L5;
template <class F>
struct AffineRound {
    const Aff<F>* src;
    const uint32_t* ent;   // the slice's first entry
    const uint32_t* total;
    uint64_t s0, slots, nbases;
    uint32_t r;
    Aff<F>* out;
    L5* acc;
};
int affine_round(const AffineRound<Fq>& a, unsigned blocks, cudaStream_t st);
int affine_round(const AffineRound<Fq2>& a, unsigned blocks, cudaStream_t st);
// A thread takes at least kAffMinPairs pairs, and a launch at most the blocks
// the device holds at once, so that the inversions are shared by as many
// pairs as the size allows.
template <class F>
inline size_t affine_blocks(size_t pairs)
{
    return grid_for(pairs / kAffMinPairs, kAffThreads, sm_count() * (sizeof(F) == 32 ? kAffBlocksG1 : kAffBlocksG2));
}
// scratch of a slice: a half and a quarter of its slots as points (the odd
// and the even rounds' results, but the last's), and the products
template <class F>
struct AffineScratch {
    size_t odd, even, acc;   // bytes
    AffineScratch(size_t slots, uint32_t rounds)
    {
        odd = align_up(rounds > 1 ? slots / 2 * sizeof(Aff<F>) : 0);
        even = align_up(rounds > 2 ? slots / 4 * sizeof(Aff<F>) : 0);
        acc = align_up(rounds ? affine_blocks<F>(slots / 2) * kAffThreads * 40 : 0);
    }
    size_t bytes() const { return odd + even + acc; }
};

// points an accumulation thread adds after the rounds: its chunk in entries
// before them, at least kMinChunk
inline uint32_t acc_chunk(uint32_t chunk, uint32_t rounds)
{
    return rounds && chunk >> rounds < kMinChunk ? kMinChunk : chunk >> rounds;
}

inline uint32_t windows_for(uint32_t c) { return (255 + c - 1) / c; }
// windows of a half scalar: its top digit, with the carry, stays <= 2^(c-1)
inline uint32_t windows_glv(uint32_t c) { return (kGlvBits + 1 + c - 1) / c; }
// Sorted entries of n scalars; their numbers, and the offsets of the buckets,
// are 32 bits.  The endomorphism makes up to two entries a scalar more than
// the plain digits do (16 against 15 at c = 17), fewer at other widths.
inline uint64_t msm_entries(uint64_t n, uint32_t c, bool glv) { return n * (glv ? 2 * windows_glv(c) : windows_for(c)); }
constexpr uint64_t kMaxEntries = (uint64_t(1) << 32) - 1;

// accumulation chunk and reduction run of an MSM of n points in group g:
// cfg's values, else the tuning table's (plain bases, or tables with
// LZK_MSM_PRECOMPUTED)
inline bool msm_shared(const lzk_msm_cfg* cfg) { return cfg && (cfg->flags & LZK_MSM_PRECOMPUTED); }
inline uint32_t msm_chunk(const lzk_msm_cfg* cfg, int group, size_t n)
{
    return cfg && cfg->acc_chunk ? cfg->acc_chunk : tune_chunk(group, n, msm_shared(cfg));
}
inline uint32_t msm_run(const lzk_msm_cfg* cfg, int group, size_t n)
{
    return cfg && cfg->reduce_run ? cfg->reduce_run : tune_run(group, n, msm_shared(cfg));
}

template <class Gp>
inline void plan_msm(MsmPlan& p, size_t n, uint32_t c, bool shared, size_t stride, uint32_t chunk = kDefaultChunk,
                     uint32_t run = kDefaultRun, uint32_t rounds = 0, bool presorted = false, bool glv = false)
{
    using X = XYZZ<typename Gp::F>;
    using A = Aff<typename Gp::F>;
    p.n = n; p.c = c; p.W = glv ? windows_glv(c) : windows_for(c); p.nb = 1u << (c - 1);
    p.glv = glv;
    p.shared = shared; p.stride = stride;
    p.wb = shared ? 1 : p.W;
    p.B = p.wb * p.nb;
    p.max_entries = msm_entries(n, c, glv);
    p.run = run;
    p.rounds = rounds;
    p.max_slots = p.max_entries + (size_t)p.B * ((1u << rounds) - 1);
    p.chunk = acc_chunk(chunk, rounds);
    p.chunks = ((p.max_slots >> rounds) + p.chunk - 1) / p.chunk;
    p.slice = p.max_slots < kAffSlice ? align_up(p.max_slots, size_t(1) << rounds) : kAffSlice;
    // bucket reduction scratch: wb * max(1, nb / kLevelL) points per buffer
    // (reduce_buckets)
    size_t lvl = (size_t)p.wb * (p.nb > kLevelL ? p.nb / kLevelL : 1);
    Carver cv;
    p.o_cnt = cv.take<uint32_t>(p.B);
    p.o_off = cv.take<uint32_t>(p.B + 1);
    p.o_ent = cv.take<uint32_t>(p.max_slots && !presorted ? p.max_slots : 1);
    p.o_bsum = cv.take<X>(p.B);
    p.o_head = cv.take<X>(p.chunks ? p.chunks : 1);
    p.o_tail = cv.take<X>(p.chunks ? p.chunks : 1);
    p.o_lr0 = cv.take<X>(lvl);
    p.o_la0 = cv.take<X>(lvl);
    p.o_lr1 = cv.take<X>(lvl);
    p.o_la1 = cv.take<X>(lvl);
    p.o_scan = cv.take<uint32_t>((p.B + 4095) / 4096 + 1);
    p.o_large = cv.take<uint32_t>(p.chunks / kFixSmall + 2);   // count, then bucket ids
    p.o_phi = cv.take<A>(glv ? 2 * n : 0);
    p.o_fin = cv.take<A>(rounds ? p.max_slots >> rounds : 0);
    p.o_aff = cv.take<char>(AffineScratch<typename Gp::F>(p.slice, rounds).bytes());
    p.bytes = cv.off;
}

// counting sort of the signed digits of all scalars into bucket lists:
// cnt/off/ent as carved by plan_msm (msm_sort.cu).  With hi given, the
// scalars are scalars[0..split) followed by hi[0..n - split).
int msm_sort(const MsmPlan& p, const Fr* scalars, uint32_t* cnt, uint32_t* off, uint32_t* ent, uint32_t* bsums,
             cudaStream_t st, const Fr* hi = nullptr, size_t split = 0);
uint32_t msm_autotune(int group, size_t n, bool shared);
// Forms of an MSM: with the affine rounds and the endomorphism where they
// apply, without the rounds, without either (the least scratch).
enum MsmForm { kMsmFull, kMsmNoRounds, kMsmLean };
// A plain G1 MSM in one of the forms without rounds, and the workspace of one.
size_t msm_form_bytes(size_t n, const lzk_msm_cfg* cfg, MsmForm form);
int msm_g1_form(const Fr* scalars, const void* bases, size_t n, Jac<Fq>* out, const lzk_msm_cfg* cfg, cudaStream_t st,
                MsmForm form);

// One digit sort shared by several shifted-table MSMs over the same scalars
// (the Groth16 A, B1 and B2 queries all take the witness): sizes of its
// buffers in 32-bit words, the sort itself, and the G1 / G2 MSMs that consume
// it (msm_sort.cu, msm_g1.cu, msm_g2.cu).  The consumers must use the same
// n, window width and table level stride as the sort.
// Rounds: those of a table MSM of n points (or 0), the same for the sort and
// its consumers, since the sort pads the buckets.
inline uint32_t table_rounds(size_t n, uint32_t c) { return affine_rounds(n * (size_t)windows_for(c), size_t(1) << (c - 1), kAffFillTable); }
struct SortWords { size_t cnt, off, ent, bsums; };
SortWords msm_sort_words(size_t n, uint32_t c, size_t stride, uint32_t rounds);
// scratch of a table MSM over a shared sort
size_t msm_presorted_bytes(int group, size_t n, const lzk_msm_cfg* cfg, uint32_t rounds);
int msm_sort_scalars(const Fr* scalars, size_t n, uint32_t c, size_t stride, uint32_t* cnt, uint32_t* off,
                     uint32_t* ent, uint32_t* bsums, cudaStream_t st, uint32_t rounds);
int msm_g1_presorted(const Fr* scalars, const void* table, size_t n, Jac<Fq>* out, const lzk_msm_cfg* cfg,
                     cudaStream_t st, const uint32_t* off, const uint32_t* ent, uint32_t rounds);
int msm_g2_presorted(const Fr* scalars, const void* table, size_t n, Jac<Fq2>* out, const lzk_msm_cfg* cfg,
                     cudaStream_t st, const uint32_t* off, const uint32_t* ent, uint32_t rounds);
// A shifted-table G1 MSM whose scalars are two arrays, lo[0..n_lo) then
// hi[0..n_hi), over one table of n_lo + n_hi points per level (msm_g1.cu):
// two MSMs whose results are only ever added, done as one (one sort, one
// bucket set, one reduction).  cfg must carry a workspace.
int msm_g1_concat(const Fr* lo, size_t n_lo, const Fr* hi, size_t n_hi, const void* table, Jac<Fq>* out,
                  const lzk_msm_cfg* cfg, cudaStream_t st, uint32_t rounds);
size_t msm_concat_bytes(size_t n, const lzk_msm_cfg* cfg, uint32_t rounds);
// exclusive scan of cnt[0..B), each rounded up to a multiple of 2^rounds,
// into off[0..B], off[B] = total; bsums holds (B + 4095) / 4096 + 1 words
// (msm_sort.cu)
int scan_offsets(uint32_t* cnt, uint32_t B, uint32_t* off, uint32_t* bsums, cudaStream_t st, uint32_t rounds = 0,
                 bool cursors = false);
// All rounds of a padded list of at most max_slots slots into fin (point i is
// what slots [i 2^rounds, (i + 1) 2^rounds) sum to), a slice at a time.
template <class F>
int affine_sum(const void* bases, const uint32_t* ent, const uint32_t* total, size_t max_slots, size_t slice,
               uint32_t rounds, uint64_t nbases, char* scratch, Aff<F>* fin, cudaStream_t st)
{
    const AffineScratch<F> sz(slice, rounds);
    AffineRound<F> a{};
    a.total = total;
    a.nbases = nbases;
    a.acc = reinterpret_cast<L5*>(scratch + sz.odd + sz.even);
    for (size_t s0 = 0; s0 < max_slots; s0 += slice) {
        a.ent = ent + s0;
        a.s0 = s0;
        a.slots = max_slots - s0 < slice ? max_slots - s0 : slice;
        a.src = static_cast<const Aff<F>*>(bases);
        for (a.r = 1; a.r <= rounds; a.r++) {
            a.out = a.r == rounds ? fin + (s0 >> rounds) : reinterpret_cast<Aff<F>*>(scratch + (a.r & 1 ? 0 : sz.odd));
            LZK_TRY(affine_round(a, (unsigned)affine_blocks<F>(a.slots >> a.r), st));
            a.src = a.out;
        }
    }
    return LZK_OK;
}

// bits [lo, lo+c) of an integer of NW limbs
template <int NW>
__device__ __forceinline__ uint32_t window_bits(const uint32_t* s, uint32_t lo, uint32_t c)
{
    const uint32_t w = lo >> 5, sh = lo & 31;
    if (w >= NW) return 0;
    const uint64_t v = ((uint64_t)s[w] | ((uint64_t)(w + 1 < NW ? s[w + 1] : 0u) << 32)) >> sh;
    return (uint32_t)v & ((1u << c) - 1u);
}

// Signed-digit recoding of a magnitude: raw = bits + carry in [0, 2^c]; raw >
// 2^(c-1) is used as raw - 2^c with a carry into the next window, so that
// |digit| <= 2^(c-1).  f(w, |digit|, negative) for every non-zero digit.
template <int NW, class Fn>
__device__ __forceinline__ void for_digits(const uint32_t* s, uint32_t c, uint32_t W, bool neg, Fn f)
{
    uint32_t carry = 0;
    const uint32_t half = 1u << (c - 1);
    for (uint32_t w = 0; w < W; w++) {
        const uint32_t raw = window_bits<NW>(s, w * c, c) + carry;
        carry = raw > half ? 1u : 0u;
        const uint32_t d = carry ? (1u << c) - raw : raw;
        if (d) f(w, d, neg != (carry != 0));
    }
}
// The digits of a scalar: of itself (h = 0), or (GLV) of its two halves, f(h,
// w, |digit|, negative).
template <bool GLV, class Fn>
__device__ __forceinline__ void scalar_digits(const Fr* sc, uint32_t c, uint32_t W, Fn f)
{
    const Fr k = from_mont(ldg_elem(sc));
    if (GLV) {
        uint32_t k1[4], k2[4];
        bool n1, n2;
        glv_split(k.v, k1, n1, k2, n2);
        for_digits<4>(k1, c, W, n1, [&](uint32_t w, uint32_t d, bool neg) { f(0u, w, d, neg); });
        for_digits<4>(k2, c, W, n2, [&](uint32_t w, uint32_t d, bool neg) { f(1u, w, d, neg); });
    } else {
        for_digits<8>(k.v, c, W, false, [&](uint32_t w, uint32_t d, bool neg) { f(0u, w, d, neg); });
    }
}

// largest b in [lo, B) with off[b] >> shift <= e
__device__ __forceinline__ uint32_t bucket_of(const uint32_t* off, uint32_t lo, uint32_t B, uint32_t e, uint32_t shift)
{
    uint32_t hi = B;  // invariant: off[lo] <= e, answer in [lo, hi)
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (off[mid] >> shift <= e) lo = mid; else hi = mid;
    }
    return lo;
}

// Base record layouts (lzk_msm_cfg.base_layout):
//   LZK_BASES_AFFINE        {x, y}, infinity = (0, 0)
//   LZK_BASES_REF_G1_JAC    the reference's G1 table records, Jacobian
//                           {X, Y, Z} (96 B) normalised by pre_comp_g1 to
//                           Z = 1 (msm.cuh:48-61); Z = 0 is infinity
//   LZK_BASES_REF_G2_LANES  the reference's device G2 records: two 96-B
//                           halves {X.c0 Y.c0 Z.c0}{X.c1 Y.c1 Z.c1}
//                           (alt_bn128_t.cuh:247-256), normalised to Z = 1
template <class F, int LAYOUT>
__device__ __forceinline__ Aff<F> load_raw(const void* bases, uint32_t idx);

template <>
__device__ __forceinline__ Aff<Fq> load_raw<Fq, LZK_BASES_AFFINE>(const void* bases, uint32_t idx)
{
    return ldg_elem(reinterpret_cast<const Aff<Fq>*>(bases) + idx);
}
template <>
__device__ __forceinline__ Aff<Fq2> load_raw<Fq2, LZK_BASES_AFFINE>(const void* bases, uint32_t idx)
{
    return ldg_elem(reinterpret_cast<const Aff<Fq2>*>(bases) + idx);
}
template <>
__device__ __forceinline__ Aff<Fq> load_raw<Fq, LZK_BASES_REF_G1_JAC>(const void* bases, uint32_t idx)
{
    Jac<Fq> j = ldg_elem(reinterpret_cast<const Jac<Fq>*>(bases) + idx);
    if (j.Z.is_zero()) return Aff<Fq>{Fq::zero(), Fq::zero()};
    return Aff<Fq>{j.X, j.Y};
}
template <>
__device__ __forceinline__ Aff<Fq2> load_raw<Fq2, LZK_BASES_REF_G2_LANES>(const void* bases, uint32_t idx)
{
    const Jac<Fq>* h = reinterpret_cast<const Jac<Fq>*>(bases) + 2 * (size_t)idx;
    Jac<Fq> h0 = ldg_elem(h), h1 = ldg_elem(h + 1);
    if (h0.Z.is_zero() && h1.Z.is_zero()) return Aff<Fq2>{Fq2::zero(), Fq2::zero()};
    return Aff<Fq2>{Fq2{h0.X, h1.X}, Fq2{h0.Y, h1.Y}};
}

// An infinite intermediate point is marked by a top word no canonical
// coordinate has, so that loading x alone shows it.
__device__ __forceinline__ bool is_marker(const Fq& x) { return x.v[7] == 0xffffffffu; }
__device__ __forceinline__ bool is_marker(const Fq2& x) { return is_marker(x.c0); }
template <class F> __device__ __forceinline__ F marker();
template <> __device__ __forceinline__ Fq marker<Fq>() { Fq m = Fq::zero(); m.v[7] = 0xffffffffu; return m; }
template <> __device__ __forceinline__ Fq2 marker<Fq2>() { return {marker<Fq>(), Fq::zero()}; }
template <>
__device__ __forceinline__ Aff<Fq> load_raw<Fq, kLayoutPoints>(const void* bases, uint32_t idx)
{
    Aff<Fq> a = ldg_elem(reinterpret_cast<const Aff<Fq>*>(bases) + idx);
    return is_marker(a.x) ? Aff<Fq>{Fq::zero(), Fq::zero()} : a;
}
// the coordinates of a G2 base that this lane holds (MemOf<Fq2P>)
template <>
__device__ __forceinline__ Aff<Fq2P> load_raw<Fq2P, LZK_BASES_AFFINE>(const void* bases, uint32_t idx)
{
    const Fq* q = reinterpret_cast<const Fq*>(reinterpret_cast<const Aff<Fq2>*>(bases) + idx) + (threadIdx.x & 1);
    return {{ldg_elem(q)}, {ldg_elem(q + 2)}};
}
template <>
__device__ __forceinline__ Aff<Fq2P> load_raw<Fq2P, kLayoutPoints>(const void* bases, uint32_t idx)
{
    Aff<Fq2P> a = load_raw<Fq2P, LZK_BASES_AFFINE>(bases, idx);
    if (__shfl_sync(Fq2P::mask(), a.x.c.v[7], threadIdx.x & 30) == 0xffffffffu) a = {Fq2P::zero(), Fq2P::zero()};
    return a;
}
template <>
__device__ __forceinline__ Aff<Fq2P> load_raw<Fq2P, LZK_BASES_REF_G2_LANES>(const void* bases, uint32_t idx)
{
    const Jac<Fq> h = ldg_elem(reinterpret_cast<const Jac<Fq>*>(bases) + 2 * (size_t)idx + (threadIdx.x & 1));
    if (Fq2P{h.Z}.is_zero()) return {Fq2P::zero(), Fq2P::zero()};
    return {{h.X}, {h.Y}};
}

template <class F, int LAYOUT>
__device__ __forceinline__ Aff<F> load_base(const void* bases, uint32_t v)
{
    Aff<F> p = load_raw<F, LAYOUT>(bases, v & 0x7fffffffu);
    if (v & 0x80000000u) { if (!aff_is_inf(p)) p.y = neg(p.y); }
    return p;
}

// The work of one accumulation thread, chunk t (k_accumulate below; the
// persistent batch kernel runs it too).  The list is the sorted entries, or
// (kLayoutPoints) the points that `shift` affine rounds left of them.
template <class F, int LAYOUT>
__device__ __forceinline__ void accumulate_chunk(uint64_t t, const void* __restrict__ bases,
                                                 const uint32_t* __restrict__ ent, const uint32_t* __restrict__ off,
                                                 uint32_t B, size_t chunks, uint32_t chunk, uint32_t shift,
                                                 uint64_t nbases, XYZZm<F>* __restrict__ bsum,
                                                 XYZZm<F>* __restrict__ head, XYZZm<F>* __restrict__ tail)
{
    (void)nbases;   // the base records behind the entries (debug checks)
    if (t >= chunks) return;
    uint32_t T = off[B] >> shift;
    uint64_t cs64 = t * chunk;
    if (cs64 >= T) return;
    uint32_t cs = (uint32_t)cs64, ce = (uint32_t)min((uint64_t)cs + chunk, (uint64_t)T);
    uint32_t b = bucket_of(off, 0, B, cs, shift);
    uint32_t bbeg = off[b] >> shift, bend = off[b + 1] >> shift;
    XYZZ<F> acc = xyzz_inf<F>();
    for (uint32_t e = cs; e < ce; e++) {
        if (e == bend) {
            // bucket b finished inside this chunk
            if (bbeg < cs) st_pt<F>(head + t, acc); else st_pt<F>(bsum + b, acc);
            // almost always the next bucket (at the prover's width a bucket
            // holds about 240 entries): one offset load instead of a binary
            // search of 16 dependent loads, which measured 0.9 % (G1) and
            // 1.3 % (G2) faster; searched only past an empty bucket.  Since
            // e < off[B], b + 1 < B and off[b + 2] exists.
            if (!LZK_CHECK(b + 2 <= B, 3)) return;
            bbeg = bend;
            bend = off[b + 2] >> shift;
            b = b + 1;
            if (bend <= e) {
                b = bucket_of(off, b + 1, B, e, shift);
                bbeg = off[b] >> shift; bend = off[b + 1] >> shift;
            }
            acc = xyzz_inf<F>();
        }
        const uint32_t v = LAYOUT == kLayoutPoints ? e : ent[e];
        if (!LZK_CHECK((v & 0x7fffffffu) < nbases, 2)) continue;
        acc = xyzz_madd(acc, load_base<F, LAYOUT>(bases, v));
    }
    bool began_before = bbeg < cs, cont_after = bend > ce;
    if (began_before) st_pt<F>(head + t, acc);
    else if (cont_after) st_pt<F>(tail + t, acc);
    else st_pt<F>(bsum + b, acc);
}
// 128-thread blocks; at most 168 registers for G1 and for G2 over two lanes (3
// blocks = 12 warps per SM) and 255 for whole G2 points (2 blocks).  With the
// products on the FP64 pipe the tighter register bounds make the product calls
// spill: G1 at 3 blocks/SM measured 6 % faster than at 5 (which matched 4 and
// 6), whole G2 points at 2 blocks 10 % faster than at 3 and 16 % than at 4.
template <class F, int LAYOUT>
__global__ void __launch_bounds__(128, sizeof(F) == 32 ? 3 : 2) k_accumulate(const void* __restrict__ bases, const uint32_t* __restrict__ ent,
                                                    const uint32_t* __restrict__ off, uint32_t B, size_t chunks,
                                                    uint32_t chunk, uint32_t shift, uint64_t nbases,
                                                    XYZZm<F>* __restrict__ bsum, XYZZm<F>* __restrict__ head,
                                                    XYZZm<F>* __restrict__ tail)
{
    accumulate_chunk<F, LAYOUT>(gtid() / MemOf<F>::lanes, bases, ent, off, B, chunks, chunk, shift, nbases, bsum, head, tail);
}

// The accumulation of a list without affine rounds.  G2 points over two lanes
// halve a chunk's chain but issue a quarter more: for lists with fewer chunks
// than the device has warps to hide the latency of.  Over reference tables of
// 16-bit windows, chunk 32, whole MSM: 4000 points (2000 chunks) 1035 us with two
// lanes, 1057 whole; 16000 (8000) 1002 and 996; 32000 1142 and 1030; 262144
// 3785 and 3106.
constexpr size_t kWholeG2Chunks = 4096;
template <class F, int LAYOUT>
inline void accumulate_plain(const void* bases, const uint32_t* ent, const uint32_t* off, uint32_t B, size_t chunks,
                             uint32_t chunk, uint64_t nbases, XYZZ<F>* bsum, XYZZ<F>* head, XYZZ<F>* tail, cudaStream_t st)
{
    using K = typename LaneOf<F>::T;
    constexpr uint32_t LP = MemOf<K>::lanes;
    if (LP == 1 || chunks >= kWholeG2Chunks)
        k_accumulate<F, LAYOUT><<<grid_for(chunks, 128), 128, 0, st>>>(bases, ent, off, B, chunks, chunk, 0, nbases, bsum, head, tail);
    else
        k_accumulate<K, LAYOUT><<<grid_for(chunks * LP, 128), 128, 0, st>>>(bases, ent, off, B, chunks, chunk, 0, nbases, bsum, head, tail);
    note_launch();
}

template <class F>
__device__ __forceinline__ void fixup_items(const uint32_t* __restrict__ off, uint32_t B, uint32_t chunk, uint32_t shift,
                        uint64_t chunks, XYZZm<F>* __restrict__ bsum, const XYZZm<F>* __restrict__ head, const XYZZm<F>* __restrict__ tail,
                        uint32_t* __restrict__ large)
{
    (void)chunks;
    for (uint64_t b = gtid() / MemOf<F>::lanes; b < B; b += gstride() / MemOf<F>::lanes) {
        uint32_t s = off[b] >> shift, e = off[b + 1] >> shift;
        if (s == e) continue;
        uint32_t c0 = s / chunk, c1 = (e - 1) / chunk;
        if (!LZK_CHECK(c1 < chunks, 4)) continue;
        if (c0 == c1) continue;
        if (c1 - c0 > kFixSmall) {
            if (MemOf<F>::lanes == 1 || !(threadIdx.x & 1)) large[1 + atomicAdd(large, 1u)] = (uint32_t)b;
            continue;
        }
        XYZZ<F> acc = ld_pt<F>(tail + c0);
        for (uint32_t c = c0 + 1; c <= c1; c++) acc = xyzz_add_cold(acc, ld_pt<F>(head + c));
        st_pt<F>(bsum + b, acc);
    }
}
template <class F>
__global__ void k_fixup(const uint32_t* __restrict__ off, uint32_t B, uint32_t chunk, uint32_t shift, uint64_t chunks,
                        XYZZm<F>* __restrict__ bsum, const XYZZm<F>* __restrict__ head, const XYZZm<F>* __restrict__ tail,
                        uint32_t* __restrict__ large)
{
    fixup_items<F>(off, B, chunk, shift, chunks, bsum, head, tail, large);
}

// One block per listed bucket: strided partial sums, then a tree in shared
// memory.  Partial q of bucket b is tail[c0] (q = 0) or head[c0 + q].
// (a point of shared memory for every point's lanes of the block at sm; the persistent batch kernel
// runs it too)
template <class F>
__device__ __forceinline__ void fixup_large_items(const uint32_t* __restrict__ off, uint32_t chunk, uint32_t shift,
                                                  XYZZm<F>* __restrict__ bsum, const XYZZm<F>* __restrict__ head,
                                                  const XYZZm<F>* __restrict__ tail, const uint32_t* __restrict__ large,
                                                  XYZZm<F>* sm)
{
    const uint32_t nl = large[0], me = threadIdx.x / MemOf<F>::lanes, all = blockDim.x / MemOf<F>::lanes;
    for (uint32_t idx = blockIdx.x; idx < nl; idx += gridDim.x) {
        uint32_t b = large[1 + idx];
        uint32_t c0 = (off[b] >> shift) / chunk, c1 = ((off[b + 1] >> shift) - 1) / chunk;
        uint32_t np = c1 - c0 + 1;
        XYZZ<F> acc = xyzz_inf<F>();
        for (uint32_t q = me; q < np; q += all)
            acc = xyzz_add_cold(acc, ld_pt<F>(q ? head + c0 + q : tail + c0));
        st_pt<F>(sm + me, acc);
        __syncthreads();
        for (uint32_t h = all / 2; h > 0; h >>= 1) {
            if (me < h) st_pt<F>(sm + me, xyzz_add_cold(ld_pt<F>(sm + me), ld_pt<F>(sm + me + h)));
            __syncthreads();
        }
        if (me == 0) st_pt<F>(bsum + b, ld_pt<F>(sm));
        __syncthreads();
    }
}
template <class F>
__global__ void k_fixup_large(const uint32_t* __restrict__ off, uint32_t chunk, uint32_t shift, XYZZm<F>* __restrict__ bsum,
                              const XYZZm<F>* __restrict__ head, const XYZZm<F>* __restrict__ tail,
                              const uint32_t* __restrict__ large)
{
    extern __shared__ uint4 fx_raw[];
    fixup_large_items<F>(off, chunk, shift, bsum, head, tail, large, reinterpret_cast<XYZZm<F>*>(fx_raw));
}

// Warp shuffles of whole points
template <class F>
__device__ __forceinline__ XYZZ<F> shfl_down_pt(const XYZZ<F>& x, uint32_t d)
{
    XYZZ<F> r;
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&x);
    uint32_t* o = reinterpret_cast<uint32_t*>(&r);
    _Pragma("unroll") for (int i = 0; i < (int)(sizeof(XYZZ<F>) / 4); i++) o[i] = __shfl_down_sync(0xffffffffu, s[i], d * MemOf<F>::lanes);
    return r;
}
template <class F>
__device__ __forceinline__ XYZZ<F> shfl_xor_pt(const XYZZ<F>& x, uint32_t m)
{
    XYZZ<F> r;
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&x);
    uint32_t* o = reinterpret_cast<uint32_t*>(&r);
    _Pragma("unroll") for (int i = 0; i < (int)(sizeof(XYZZ<F>) / 4); i++) o[i] = __shfl_xor_sync(0xffffffffu, s[i], m * MemOf<F>::lanes);
    return r;
}
template <class F>
__device__ __forceinline__ XYZZ<F> shfl_pt(const XYZZ<F>& x, uint32_t lane)
{
    XYZZ<F> r;
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&x);
    uint32_t* o = reinterpret_cast<uint32_t*>(&r);
    _Pragma("unroll") for (int i = 0; i < (int)(sizeof(XYZZ<F>) / 4); i++) o[i] = __shfl_sync(0xffffffffu, s[i], lane);
    return r;
}

// the warp's first point, whole, in every lane
template <class F>
__device__ __forceinline__ XYZZm<F> whole_pt(const XYZZ<F>& x)
{
    if constexpr (MemOf<F>::lanes == 2) {
        return {{shfl_elem(x.X.c, 0), shfl_elem(x.X.c, 1)}, {shfl_elem(x.Y.c, 0), shfl_elem(x.Y.c, 1)},
                {shfl_elem(x.ZZ.c, 0), shfl_elem(x.ZZ.c, 1)}, {shfl_elem(x.ZZZ.c, 0), shfl_elem(x.ZZZ.c, 1)}};
    } else {
        return shfl_pt(x, 0);
    }
}

// ---------------------------- bucket reduction ----------------------------
// Per bucket set (one per window for plain bases, one for all windows with a
// shifted-copy table) of m = 2^(c-1) buckets B_0..B_{m-1}, bucket k holding
// digit k + 1, the weighted sum W = sum_k (k+1) B_k.  With tiles of L
// buckets and P = m / L tiles,
//   W = sum_u t_u + L sum_u u R_u = T + sum_{i < log P} 2^(i + log L) G_i,
// where R_u is the sum of tile u, t_u = sum_j (j+1) B_{uL+j} its locally
// weighted sum, T = sum_u t_u and G_i = sum of the R_u with bit i of u set
// (bit slices of the tile index).  Four launches, each over the items of
// any number of jobs (reduce_jobs):
//   k_red_tile     one warp per tile (below);
//   k_red_slices   one warp per 32 members of one of the 1 + log P sums T,
//                  G_0, G_1, ... (xor-shuffle tree);
//   k_red_scale    one warp per sum: fold its partials, double it
//                  i + log L times (warp-uniform doublings);
//   k_red_combine  one warp per set: add the scaled sums.
// For m = 2^16 the longest chain is 19 + 5 + 6 + 15 doublings + 5 dependent
// point operations; a ladder of 32-bucket levels with the weights carried by
// doublings at every level needs about twice that.  Empty buckets
// (off[k] == off[k+1]) read as the point at infinity.
//
// k_red_tile: lane j of a tile holds the run of r consecutive buckets
// jr .. jr + r - 1 (r = 4 for m >= 128, L = 32 r; smaller sets take r = 2 or
// 1 and L = m).  The lane forms the run's sum s_j and its locally weighted
// sum t_j = sum_i (i+1) B_{jr+i} by running sums (two additions per
// bucket), a shuffle suffix scan gives S_j = sum_{j'>=j} s_j', and since the
// tile-local weight of bucket jr + i is jr + i + 1,
//   R_u = S_0,   t_u = sum_j (t_j + r [j >= 1] S_j).
// About 4.75 additions per bucket for r = 4, against 10 for a warp scan over
// single buckets (r = 1).
struct RedShape {
    uint32_t r, L, lgL, P, lg;   // buckets per lane run, tile size, log2 L, tiles per set, log2 P
    uint32_t cT, cG, NP, NS;     // chunks of T, chunks of each G_i, partials and sums per set
};
// run: requested buckets per lane run (a power of two); a set too small
// for 32 lanes of such runs takes shorter runs, down to single buckets
// lanes: points a warp holds.  16 (two lanes a point) take runs of two at
// least, so that no set has more tiles than the scratch is sized for.
inline RedShape red_shape(uint32_t m, uint32_t run, uint32_t lanes)
{
    RedShape s;
    const uint32_t least = 32 / lanes;
    s.r = run > least ? run : least;
    while (s.r > least && lanes * s.r > m) s.r >>= 1;
    while (s.r > 1 && s.r > m) s.r >>= 1;
    s.L = m < lanes * s.r ? m : lanes * s.r;
    s.lgL = 0; while ((1u << s.lgL) < s.L) s.lgL++;
    s.P = m / s.L;
    s.lg = 0; while ((1u << s.lg) < s.P) s.lg++;
    s.cT = (s.P + lanes - 1) / lanes;
    s.cG = (s.P / 2 + lanes - 1) / lanes;
    s.NP = s.cT + s.lg * s.cG;
    s.NS = 1 + s.lg;
    return s;
}

// member v of slice i: the v-th tile index with bit i set
__device__ __forceinline__ uint32_t slice_member(uint32_t v, uint32_t i)
{
    return ((v >> i) << (i + 1)) | (1u << i) | (v & ((1u << i) - 1));
}

// One reduction job: wb sets of m buckets (bsum / off indexed w m + k) into
// win[0..wb), with scratch R, T, part, scaled of its own (at least wb * P
// points each; NP, NS <= P), so that the jobs of several window widths (a
// batch plan's width groups) run in the same launches.  s_* is the job's
// first item in each launch's item space (the items of all jobs laid end to
// end: tiles wb P, slice partials wb NP, sums wb NS, sets wb).
template <class F>
struct RedJob {
    const XYZZm<F>* bsum;
    const uint32_t* off;
    XYZZm<F> *R, *T, *part, *scaled, *win;
    uint32_t wb, m;
    RedShape sh;
    uint64_t s_tile, s_np, s_ns, s_w;
};
constexpr uint32_t kMaxRedJobs = 20;   // a kernel parameter of about 3 KB
template <class F>
struct RedJobs {
    uint32_t count;
    RedJob<F> g[kMaxRedJobs];
};

// the job whose items include `item` (jobs in item order)
template <class F>
__device__ __forceinline__ uint32_t red_job_of(const RedJobs<F>& jobs, uint64_t item, uint64_t RedJob<F>::*start)
{
    uint32_t j = 0;
    while (j + 1 < jobs.count && item >= jobs.g[j + 1].*start) j++;
    return j;
}

template <class F>
__device__ __forceinline__ void red_tile_items(const RedJobs<F>& jobs, uint64_t total)
{
    constexpr uint32_t LP = MemOf<F>::lanes, NL = 32 / LP;
    const uint32_t lane = (threadIdx.x & 31) / LP;
    for (uint64_t item = gtid() >> 5; item < total; item += gstride() >> 5) {
        const RedJob<F>& J = jobs.g[red_job_of(jobs, item, &RedJob<F>::s_tile)];
        const uint64_t tile = item - J.s_tile;
        const uint32_t L = J.sh.L, r = J.sh.r;
        const uint32_t nl = L / r;   // active lanes
        XYZZ<F> s = xyzz_inf<F>(), t = xyzz_inf<F>();
        if (lane < nl) {
            const size_t k0 = (size_t)tile * L + (size_t)lane * r;   // = w m + u L + j r
            for (int i = (int)r - 1; i >= 0; i--) {
                size_t k = k0 + (uint32_t)i;
                if (J.off[k] != J.off[k + 1]) s = xyzz_add_cold(s, ld_pt<F>(J.bsum + k));
                t = xyzz_add_cold(t, s);
            }
        }
        XYZZ<F> S = s;
        for (uint32_t d = 1; d < nl; d <<= 1) {
            XYZZ<F> o = shfl_down_pt(S, d);
            if (lane + d < nl) S = xyzz_add_cold(S, o);
        }
        XYZZ<F> U = (lane >= 1 && lane < nl) ? S : xyzz_inf<F>();
        for (uint32_t q = r; q > 1; q >>= 1) U = xyzz_dbl_cold(U);
        XYZZ<F> V = xyzz_add_cold(t, U);
        for (uint32_t d = nl >> 1; d > 0; d >>= 1) V = xyzz_add_cold(V, shfl_xor_pt(V, d));
        if (lane == 0) {
            st_pt<F>(J.R + tile, S);
            st_pt<F>(J.T + tile, V);
        }
    }
}
template <class F>
__global__ void __launch_bounds__(128) k_red_tile(const __grid_constant__ RedJobs<F> jobs, uint64_t total)
{
    red_tile_items<F>(jobs, total);
}


template <class F>
__device__ __forceinline__ void red_slices_items(const RedJobs<F>& jobs, uint64_t total)
{
    constexpr uint32_t LP = MemOf<F>::lanes, NL = 32 / LP;
    const uint32_t lane = (threadIdx.x & 31) / LP;
    for (uint64_t item = gtid() >> 5; item < total; item += gstride() >> 5) {
        const RedJob<F>& J = jobs.g[red_job_of(jobs, item, &RedJob<F>::s_np)];
        const RedShape& sh = J.sh;
        const uint64_t g = item - J.s_np;
        uint32_t w = (uint32_t)(g / sh.NP), q = (uint32_t)(g % sh.NP);
        const size_t base = (size_t)w * sh.P;
        XYZZ<F> x = xyzz_inf<F>();
        if (q < sh.cT) {
            uint32_t v = q * NL + lane;
            if (v < sh.P) x = ld_pt<F>(J.T + base + v);
        } else {
            uint32_t i = (q - sh.cT) / sh.cG, v = ((q - sh.cT) % sh.cG) * NL + lane;
            if (v < sh.P / 2) x = ld_pt<F>(J.R + base + slice_member(v, i));
        }
        for (uint32_t d = NL / 2; d > 0; d >>= 1) x = xyzz_add_cold(x, shfl_xor_pt(x, d));
        if (lane == 0) st_pt<F>(J.part + g, x);
    }
}
template <class F>
__global__ void __launch_bounds__(128) k_red_slices(const __grid_constant__ RedJobs<F> jobs, uint64_t total)
{
    red_slices_items<F>(jobs, total);
}

template <class F>
__device__ __forceinline__ void red_scale_items(const RedJobs<F>& jobs, uint64_t total)
{
    constexpr uint32_t LP = MemOf<F>::lanes, NL = 32 / LP;
    const uint32_t lane = (threadIdx.x & 31) / LP;
    for (uint64_t item = gtid() >> 5; item < total; item += gstride() >> 5) {
        const RedJob<F>& J = jobs.g[red_job_of(jobs, item, &RedJob<F>::s_ns)];
        const RedShape& sh = J.sh;
        const uint64_t g = item - J.s_ns;
        uint32_t w = (uint32_t)(g / sh.NS), s = (uint32_t)(g % sh.NS);
        uint32_t first = s == 0 ? 0 : sh.cT + (s - 1) * sh.cG, cnt = s == 0 ? sh.cT : sh.cG;
        const XYZZm<F>* src = J.part + (size_t)w * sh.NP + first;
        XYZZ<F> x = xyzz_inf<F>();
        for (uint32_t c = lane; c < cnt; c += NL) x = xyzz_add_cold(x, ld_pt<F>(src + c));
        for (uint32_t d = NL / 2; d > 0; d >>= 1) x = xyzz_add_cold(x, shfl_xor_pt(x, d));
        // lanes may hold different representations of the sum (an addition
        // with swapped operands negates Y and ZZZ); the warp-uniform
        // doublings need one
        XYZZm<F> y = whole_pt(x);
        uint32_t dbls = s == 0 ? 0 : s - 1 + sh.lgL;
        for (uint32_t d = 0; d < dbls; d++) y = xyzz_dbl_warp(y);
        if ((threadIdx.x & 31) == 0) st_elem(J.scaled + g, y);
    }
}
template <class F>
__global__ void __launch_bounds__(128) k_red_scale(const __grid_constant__ RedJobs<F> jobs, uint64_t total)
{
    red_scale_items<F>(jobs, total);
}

template <class F>
__device__ __forceinline__ void red_combine_items(const RedJobs<F>& jobs, uint64_t total)
{
    constexpr uint32_t LP = MemOf<F>::lanes, NL = 32 / LP;
    const uint32_t lane = (threadIdx.x & 31) / LP;
    for (uint64_t item = gtid() >> 5; item < total; item += gstride() >> 5) {
        const RedJob<F>& J = jobs.g[red_job_of(jobs, item, &RedJob<F>::s_w)];
        const uint64_t w = item - J.s_w;
        const uint32_t NS = J.sh.NS;
        XYZZ<F> x = xyzz_inf<F>();
        for (uint32_t c = lane; c < NS; c += NL) x = xyzz_add_cold(x, ld_pt<F>(J.scaled + w * NS + c));
        for (uint32_t d = NL / 2; d > 0; d >>= 1) x = xyzz_add_cold(x, shfl_xor_pt(x, d));
        if (lane == 0) st_pt<F>(J.win + w, x);
    }
}
template <class F>
__global__ void __launch_bounds__(128) k_red_combine(const __grid_constant__ RedJobs<F> jobs, uint64_t total)
{
    red_combine_items<F>(jobs, total);
}

// Scratch points each of R, T, part and scaled needs for wb sets of m
// buckets (any run: P <= max(1, m / kLevelL), NP, NS <= P).
inline size_t red_scratch_points(uint32_t wb, uint32_t m) { return (size_t)wb * (m > kLevelL ? m / kLevelL : 1); }

template <class F>
RedJob<F> red_job(const XYZZm<F>* bsum, const uint32_t* off, uint32_t wb, uint32_t m, uint32_t run, XYZZm<F>* R,
                  XYZZm<F>* T, XYZZm<F>* part, XYZZm<F>* scaled, XYZZm<F>* win)
{
    RedJob<F> j{};
    j.bsum = bsum; j.off = off; j.R = R; j.T = T; j.part = part; j.scaled = scaled; j.win = win;
    j.wb = wb; j.m = m;
    j.sh = red_shape(m, run, 32 / MemOf<F>::lanes);
    return j;
}

// The weighted sums of every job, four launches for all of them (in rounds
// of kMaxRedJobs jobs).  A job's win may alias its R.
template <class F>
int reduce_jobs(RedJob<F>* jv, size_t n, cudaStream_t st)
{
    for (size_t b = 0; b < n; b += kMaxRedJobs) {
        RedJobs<F> jobs{};
        jobs.count = (uint32_t)(n - b < kMaxRedJobs ? n - b : kMaxRedJobs);
        uint64_t tiles = 0, nps = 0, nss = 0, sets = 0;
        for (uint32_t i = 0; i < jobs.count; i++) {
            RedJob<F> j = jv[b + i];
            j.s_tile = tiles; j.s_np = nps; j.s_ns = nss; j.s_w = sets;
            tiles += (uint64_t)j.wb * j.sh.P;
            nps += (uint64_t)j.wb * j.sh.NP;
            nss += (uint64_t)j.wb * j.sh.NS;
            sets += j.wb;
            jobs.g[i] = j;
        }
        k_red_tile<F><<<grid_for(tiles * 32, 128), 128, 0, st>>>(jobs, tiles); note_launch();
        k_red_slices<F><<<grid_for(nps * 32, 128), 128, 0, st>>>(jobs, nps); note_launch();
        k_red_scale<F><<<grid_for(nss * 32, 128), 128, 0, st>>>(jobs, nss); note_launch();
        k_red_combine<F><<<grid_for(sets * 32, 128), 128, 0, st>>>(jobs, sets); note_launch();
        LZK_TRY(launch_status());
    }
    return LZK_OK;
}

// W_w of wb sets of m buckets (bsum / off indexed w m + k) into win[0..wb).
// Scratch: R, T, part, scaled of red_scratch_points(wb, m) points each.  win
// may alias R.
template <class F>
int reduce_buckets(const XYZZm<F>* bsum, const uint32_t* off, uint32_t wb, uint32_t m, XYZZm<F>* R, XYZZm<F>* T,
                   XYZZm<F>* part, XYZZm<F>* scaled, XYZZm<F>* win, cudaStream_t st, uint32_t run = kDefaultRun)
{
    RedJob<F> j = red_job<F>(bsum, off, wb, m, run, R, T, part, scaled, win);
    return reduce_jobs<F>(&j, 1, st);
}

// Horner over the bucket sets' weighted sums (plain bases), or the
// conversion of the one set's sum (shifted-copy table): one warp, with
// warp-uniform point operations.  Launched as <<<1, 32>>>.
template <class F>
__global__ void k_finish(const XYZZ<F>* __restrict__ win, uint32_t windows, uint32_t c, Jac<F>* out)
{
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    XYZZ<F> r = xyzz_inf<F>();
    for (int w = (int)windows - 1; w >= 0; w--) {
        if (w != (int)windows - 1)
            for (uint32_t d = 0; d < c; d++) r = xyzz_dbl_warp(r);
        r = xyzz_add_warp(r, ld_elem(win + w));
    }
    Jac<F> j = xyzz_to_jac_warp(r);
    if (threadIdx.x == 0) st_elem(out, j);
}

template <class F>
__global__ void k_write_inf(Jac<F>* out)
{
    if (gtid() == 0) st_elem(out, Jac<F>{F::zero(), F::one(), F::zero()});
}

// Plain G1 bases are doubled by the endomorphism: half the windows, bucket
// sets and serial doublings for the same additions, where the entries can be
// numbered and the doubled bases keep their sign bit.  (G2 has none that holds
// for points outside the prime-order subgroup; a table needs none of these.)
inline bool msm_glv(int group, size_t n, uint32_t c, bool shared)
{
    return group == 1 && !shared && n < (size_t(1) << 30) && msm_entries(n, c, true) <= kMaxEntries;
}
// whether an MSM of n points can be sorted at this width, in either form
inline bool msm_width_fits(int group, size_t n, uint32_t c, bool shared)
{
    return msm_glv(group, n, c, shared) || msm_entries(n, c, false) <= kMaxEntries;
}
// affine rounds of an MSM over bases in this layout
inline uint32_t msm_rounds(int group, size_t n, uint32_t c, bool shared, uint32_t layout)
{
    const bool glv = msm_glv(group, n, c, shared);
    const size_t W = glv ? windows_glv(c) : windows_for(c);
    return layout == LZK_BASES_AFFINE || glv ? affine_rounds(msm_entries(n, c, glv), (shared ? 1 : W) << (c - 1),
                                                             shared ? kAffFillTable : kAffFillPlain)
                                           : 0;
}

// out[i] = base i, out[n + i] = phi(base i)
template <int LAYOUT>
__global__ void k_glv_bases(const void* __restrict__ bases, size_t n, Aff<Fq>* __restrict__ out)
{
    for (uint64_t i = gtid(); i < n; i += gstride()) {
        Aff<Fq> p = load_raw<Fq, LAYOUT>(bases, (uint32_t)i);
        st_elem(out + i, p);
        p.x = mul52(p.x, glv_beta());
        st_elem(out + n + i, p);
    }
}

// pre_off / pre_ent: bucket offsets and sorted entries of these scalars made
// earlier by msm_sort for the same n, window width and table stride (MSMs
// over the same scalars share one sort, padded for pre_rounds affine rounds);
// null = sort here.
template <class Gp>
int run_msm(const Fr* scalars, const void* bases, size_t n, Jac<typename Gp::F>* out,
                   const lzk_msm_cfg* cfg, cudaStream_t st, uint32_t c_auto,
                   const uint32_t* pre_off = nullptr, const uint32_t* pre_ent = nullptr, uint32_t pre_rounds = 0,
                   bool pre_in_ws = false, MsmForm form = kMsmFull)
{
    using F = typename Gp::F;
    using X = XYZZ<F>;
    using A = Aff<F>;
    using K = typename LaneOf<F>::T;   // coordinates in the accumulation and after it
    constexpr uint32_t LP = MemOf<K>::lanes;
    if (!out || (n && (!scalars || !bases))) return LZK_EINVAL;
    if (n >= (1ull << 31)) return LZK_EINVAL;
    uint32_t flags = cfg ? cfg->flags : 0u;
    uint32_t layout = cfg ? cfg->base_layout : (uint32_t)LZK_BASES_AFFINE;
    uint32_t ref_layout = sizeof(F) == 32 ? LZK_BASES_REF_G1_JAC : LZK_BASES_REF_G2_LANES;
    if (layout != LZK_BASES_AFFINE && layout != ref_layout) return LZK_EINVAL;
    bool shared = (flags & LZK_MSM_PRECOMPUTED) != 0;
    uint32_t c = (cfg && cfg->window_bits) ? cfg->window_bits : c_auto;
    if (c < 2 || c > 24) return LZK_EINVAL;
    size_t stride = shared ? cfg->level_stride : 0;
    if (shared) {
        if (!cfg->window_bits) return LZK_EINVAL;
        if (cfg->precomp_windows < windows_for(c) || stride < n) return LZK_EINVAL;
        if ((size_t)windows_for(c) * stride >= (1ull << 31)) return LZK_EINVAL;
    }
    if (n == 0) {
        k_write_inf<F><<<1, 32, 0, st>>>(out); note_launch();
        return launch_status();
    }
    const int group = sizeof(F) == 32 ? 1 : 2;
    if (!msm_width_fits(group, n, c, shared)) return LZK_EINVAL;
    uint32_t chunk = msm_chunk(cfg, group, n), run = msm_run(cfg, group, n);
    if (!tune_valid(LZK_TUNE_MSM_CHUNK, chunk) || !tune_valid(LZK_TUNE_MSM_REDUCE_RUN, run)) return LZK_EINVAL;
    MsmPlan p;
    plan_msm<Gp>(p, n, c, shared, stride, chunk, run,
                 form != kMsmFull ? 0 : pre_off ? pre_rounds : msm_rounds(group, n, c, shared, layout),
                 pre_off && !pre_in_ws, form != kMsmLean && msm_glv(group, n, c, shared));
    void* tr_all = trace_begin(sizeof(F) == 32 ? "msm_g1" : "msm_g2", st);
    Scratch ws;
    int got = ws.acquire(p.bytes, cfg ? cfg->workspace : nullptr, cfg ? cfg->workspace_bytes : 0, st);
    if (got != LZK_OK && (p.rounds || p.glv) && !pre_off && msm_entries(n, c, false) <= kMaxEntries) {
        // too little scratch for the affine rounds and the doubled bases: XYZZ
        // additions alone
        plan_msm<Gp>(p, n, c, shared, stride, chunk, run);
        got = ws.acquire(p.bytes, cfg ? cfg->workspace : nullptr, cfg ? cfg->workspace_bytes : 0, st);
    }
    LZK_TRY(got);
    char* base = ws.base;
    uint32_t* cnt = reinterpret_cast<uint32_t*>(base + p.o_cnt);
    uint32_t* off_ws = reinterpret_cast<uint32_t*>(base + p.o_off);
    uint32_t* ent_ws = reinterpret_cast<uint32_t*>(base + p.o_ent);
    const uint32_t* off = pre_off ? pre_off : off_ws;
    const uint32_t* ent = pre_ent ? pre_ent : ent_ws;
    X* bsum = reinterpret_cast<X*>(base + p.o_bsum);
    X* head = reinterpret_cast<X*>(base + p.o_head);
    X* tail = reinterpret_cast<X*>(base + p.o_tail);
    X* lr[2] = {reinterpret_cast<X*>(base + p.o_lr0), reinterpret_cast<X*>(base + p.o_lr1)};
    X* la[2] = {reinterpret_cast<X*>(base + p.o_la0), reinterpret_cast<X*>(base + p.o_la1)};

    uint32_t* bsums = reinterpret_cast<uint32_t*>(base + p.o_scan);
    uint32_t* large = reinterpret_cast<uint32_t*>(base + p.o_large);
    if (!pre_off) {
        void* tr_sort = trace_begin(sizeof(F) == 32 ? "msm_g1_sort" : "msm_g2_sort", st);
        LZK_TRY(msm_sort(p, scalars, cnt, off_ws, ent_ws, bsums, st));
        trace_end(tr_sort, st);
    }
    if constexpr (sizeof(F) == 32) {
        if (p.glv) {
            A* phi = reinterpret_cast<A*>(base + p.o_phi);
            const unsigned g = grid_for(n, 128, sm_count() * 16);
            if (layout == LZK_BASES_AFFINE) k_glv_bases<LZK_BASES_AFFINE><<<g, 128, 0, st>>>(bases, n, phi);
            else k_glv_bases<LZK_BASES_REF_G1_JAC><<<g, 128, 0, st>>>(bases, n, phi);
            note_launch();
            bases = phi;
            layout = LZK_BASES_AFFINE;
        }
    }
    void* tr = trace_begin(sizeof(F) == 32 ? "msm_g1_accumulate" : "msm_g2_accumulate", st);
    {
        unsigned g = grid_for(p.chunks * LP, 128);
        // base records the entries may name: the whole table, or the n bases
        const uint64_t nbases = shared ? (uint64_t)cfg->precomp_windows * stride : (uint64_t)n * (p.glv ? 2 : 1);
        constexpr int REF = sizeof(F) == 32 ? (int)LZK_BASES_REF_G1_JAC : (int)LZK_BASES_REF_G2_LANES;
        if (p.rounds) {
            A* fin = reinterpret_cast<A*>(base + p.o_fin);
            LZK_TRY(affine_sum<F>(bases, ent, off + p.B, p.max_slots, p.slice, p.rounds, nbases,
                                  base + p.o_aff, fin, st));
            k_accumulate<K, kLayoutPoints><<<g, 128, 0, st>>>(fin, ent, off, p.B, p.chunks, p.chunk, p.rounds, p.max_slots >> p.rounds, bsum, head, tail); note_launch();
        } else if (layout == LZK_BASES_AFFINE) {
            accumulate_plain<F, LZK_BASES_AFFINE>(bases, ent, off, p.B, p.chunks, p.chunk, nbases, bsum, head, tail, st);
        } else {
            accumulate_plain<F, REF>(bases, ent, off, p.B, p.chunks, p.chunk, nbases, bsum, head, tail, st);
        }
    }
    trace_end(tr, st);
    void* tr_fix = trace_begin(sizeof(F) == 32 ? "msm_g1_fixup" : "msm_g2_fixup", st);
    LZK_CUDA(cudaMemsetAsync(large, 0, sizeof(uint32_t), st));
    k_fixup<K><<<grid_for((size_t)p.B * LP, 256, sm_count() * 8), 256, 0, st>>>(off, p.B, p.chunk, p.rounds, p.chunks, bsum, head, tail, large); note_launch();
    {
        constexpr unsigned fx_points = 32768 / sizeof(X);   // 32 KB of shared memory
        k_fixup_large<K><<<sm_count() * 2, fx_points * LP, fx_points * sizeof(X), st>>>(off, p.chunk, p.rounds, bsum, head, tail, large); note_launch();
    }
    trace_end(tr_fix, st);
    LZK_TRY(launch_status());

    // weighted sums per bucket set
    void* tr_red = trace_begin(sizeof(F) == 32 ? "msm_g1_reduce" : "msm_g2_reduce", st);
    X* win = lr[0];
    LZK_TRY(reduce_buckets<K>(bsum, off, p.wb, p.nb, lr[0], la[0], lr[1], la[1], win, st, p.run));
    void* tr_fin = trace_begin(sizeof(F) == 32 ? "msm_g1_finish" : "msm_g2_finish", st);
    k_finish<F><<<1, 32, 0, st>>>(win, p.wb, c, out); note_launch();
    trace_end(tr_fin, st);
    trace_end(tr_red, st);
    trace_end(tr_all, st);
    return launch_status();
}

// ------------------------- precomputed shifted bases -------------------------
template <class F>
__global__ void k_precompute(const Aff<F>* __restrict__ bases, size_t n, uint32_t c, uint32_t windows,
                             Aff<F>* __restrict__ table, size_t stride)
{
    // windows are normalised in groups of G with one inversion per group
    constexpr int G = 8;
    for (uint64_t i = gtid(); i < n; i += gstride()) {
        Aff<F> P = ldg_elem(bases + i);
        st_elem(table + i, P);
        if (aff_is_inf(P)) {
            Aff<F> z{F::zero(), F::zero()};
            for (uint32_t j = 1; j < windows; j++) st_elem(table + (size_t)j * stride + i, z);
            continue;
        }
        XYZZ<F> cur = xyzz_from_aff(P);
        for (uint32_t j0 = 1; j0 < windows; j0 += G) {
            int cntg = (int)min((uint32_t)G, windows - j0);
            XYZZ<F> pts[G];
            F pre[G];
            F acc = F::one();
            for (int k = 0; k < cntg; k++) {
                for (uint32_t d = 0; d < c; d++) cur = xyzz_dbl_cold(cur);
                pts[k] = cur;
                acc = mul(acc, mul(cur.ZZ, cur.ZZZ));
                pre[k] = acc;
            }
            F inv = inverse(acc);
            for (int k = cntg - 1; k >= 0; k--) {
                F dinv = k ? mul(inv, pre[k - 1]) : inv;  // (ZZ_k ZZZ_k)^-1
                inv = mul(inv, mul(pts[k].ZZ, pts[k].ZZZ));
                // x = X / ZZ = X * ZZZ * dinv,  y = Y / ZZZ = Y * ZZ * dinv
                Aff<F> a{mul(mul(pts[k].X, dinv), pts[k].ZZZ), mul(mul(pts[k].Y, dinv), pts[k].ZZ)};
                st_elem(table + (size_t)(j0 + k) * stride + i, a);
            }
        }
    }
}

// Jacobian -> affine, 8 points per thread with one inversion
template <class F>
__global__ void k_jac_to_aff(const Jac<F>* __restrict__ in, Aff<F>* __restrict__ out, size_t n)
{
    constexpr int G = 8;
    for (uint64_t t = gtid(); t * G < n; t += gstride()) {
        size_t b = t * G;
        int cntp = (int)((n - b) < G ? (n - b) : G);
        F pre[G];
        F acc = F::one();
        for (int k = 0; k < cntp; k++) {
            Jac<F> J = ld_elem(in + b + k);
            if (!J.Z.is_zero()) acc = mul(acc, J.Z);
            pre[k] = acc;
        }
        F inv = inverse(acc);
        for (int k = cntp - 1; k >= 0; k--) {
            Jac<F> J = ld_elem(in + b + k);
            if (J.Z.is_zero()) { st_elem(out + b + k, Aff<F>{F::zero(), F::zero()}); continue; }
            F zi = k ? mul(inv, pre[k - 1]) : inv;
            inv = mul(inv, J.Z);
            F z2 = sqr(zi);
            st_elem(out + b + k, Aff<F>{mul(J.X, z2), mul(J.Y, mul(z2, zi))});
        }
    }
}

template <class F>
int run_precompute(const Aff<F>* bases, size_t n, uint32_t c, uint32_t windows, Aff<F>* table,
                          size_t stride, cudaStream_t st)
{
    if (!bases || !table || c < 2 || c > 24 || windows == 0 || windows > 256 || stride < n) return LZK_EINVAL;
    if (n == 0) return LZK_OK;
    k_precompute<F><<<grid_for(n, 64), 64, 0, st>>>(bases, n, c, windows, table, stride); note_launch();
    return launch_status();
}

}  // namespace lzk
