// Index logic and butterflies of the two-phase NTT (see wg_ntt.cu), shared by the device
// kernels and the CPU emulation test.
#pragma once
#include <cstddef>
#include <cstdint>
#include <utility>

#include "wg_arith.cuh"
#include "wg_fp.cuh"

namespace wg {
namespace ntt {

constexpr int kMaxTile = 2048;

// One entry of the interleaved twiddle table: the twiddle and its Shoup constant (for the moduli of
// the FP64 path: the doubles w and w / q, twiddle_pair) side by side, so a butterfly fetches both
// with one 16-byte load.  Table layout per modulus:
// [forward pairs (N)][inverse pairs (N)], one order per residues-per-thread (twiddle_place).
struct alignas(16) TwPair {
    uint64_t w, ws;
};

WG_HD int pad16(int e) { return e + (e >> 4); }
WG_HD int floor_log2(unsigned x) {
#if defined(__CUDA_ARCH__)
    return 31 - __clz(x);
#else
    return 31 - __builtin_clz(x);
#endif
}
WG_HD int insert_zero(int v, int g) {
    return ((v >> g) << (g + 1)) | (v & ((1 << g) - 1));
}

// Bits handled by one round: up to EB stage bits (in processing order) plus filler bits (the
// lowest free bits) so every thread always owns 2^EB elements.  The forward transform's rounds go
// down from the highest bit in groups of EB, the last one taking what is left; the inverse's rounds
// are the same groups from the last to the first, so a thread owns the same elements in the
// inverse's last round as in the forward's first.
struct RoundPlan {
    int ns;
    int sb[4];  // stage bits, processing order
    int jb[4];  // position of each stage bit inside the EB-bit element index j
    int g[4];   // group bits ascending
};

template <int MB, bool FWD, int EB>
WG_HDC constexpr RoundPlan make_plan(int rd) {
    RoundPlan p{0, {0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}};
    const int fr = FWD ? rd : (MB + EB - 1) / EB - 1 - rd;  // the forward round with the same group
    for (int k = 0; k < EB; ++k) {
        const int b = MB - 1 - EB * fr - (FWD ? k : EB - 1 - k);
        if (b >= 0) p.sb[p.ns++] = b;
    }
    int mask = 0;
    for (int k = 0; k < p.ns; ++k) mask |= 1 << p.sb[k];
    int filled = p.ns;
    for (int b = 0; filled < EB; ++b)
        if (!((mask >> b) & 1)) {
            mask |= 1 << b;
            ++filled;
        }
    int k = 0;
    for (int b = 0; b < 32 && k < EB; ++b)
        if ((mask >> b) & 1) p.g[k++] = b;
    for (int s = 0; s < p.ns; ++s)
        for (int x = 0; x < EB; ++x)
            if (p.sb[s] == p.g[x]) p.jb[s] = x;
    return p;
}

// Geometry of one phase of an N = 2^LOGN transform.
//   EB:     a thread carries 2^EB residues through each round (3: radix-8 rounds of up to three
//           stages; 4: radix-16 rounds of up to four).  They come from device memory into the first
//           round's registers and leave from the last one's; between rounds the CTA exchanges them
//           through shared memory;
//   STAGED: the CTA first copies the twiddle pairs it will read into shared memory; otherwise
//           the rounds read them from the (L2-resident) global table directly, which leaves
//           shared memory to the data tile and admits more CTAs per SM.
//   TL:     largest tile (elements per CTA); a column-phase tile holds TL >> NB1 whole columns.
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL = kMaxTile>
struct Phase {
    static constexpr int N = 1 << LOGN;
    static constexpr int NB1 = LOGN / 2;
    static constexpr int NB2 = LOGN - NB1;
    static constexpr int MB = COLS ? NB1 : NB2;
    static constexpr int E = 1 << EB;
    static constexpr int TILE = N < TL ? N : TL;
    static constexpr int THREADS = TILE / E;
    static constexpr int SUBS = TILE >> MB;  // sub-transforms per tile
    static constexpr int OB = MB - EB;
    static constexpr int ROUNDS = (MB + EB - 1) / EB;
    static constexpr bool LAST = FWD ? !COLS : COLS;
    WG_HD static int sub_of(int t) { return COLS ? t % SUBS : t >> OB; }
    WG_HD static int o_of(int t) { return COLS ? t / SUBS : t & ((1 << OB) - 1); }
    // Twiddle pairs one CTA reads (staged in shared memory when STAGED): the column phase reads
    // table entries [0, 2^NB1); the row phase reads, for row-stage k, SUBS * 2^k contiguous
    // entries.
    static constexpr int TW = COLS ? (1 << NB1) : (TILE - SUBS);
    static_assert(MB >= EB, "transform too small for this round radix");
    static_assert(EB >= 2 && EB <= 4, "rounds of 4, 8 or 16 residues per thread");
};

// Table index of staged twiddle t (see Phase::TW).  Row-stage k occupies staged entries
// [SUBS (2^k - 1), SUBS (2^(k+1) - 1)) and maps to table entries starting at
// 2^(NB1 + k) + tile * SUBS * 2^k.
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL = kMaxTile>
WG_HD size_t twiddle_src(int tile, int t) {
    using P = Phase<LOGN, FWD, COLS, EB, STAGED, TL>;
    if (COLS) return (size_t)t;
    const int k = floor_log2((unsigned)(t / P::SUBS + 1));
    const int off = P::SUBS * ((1 << k) - 1);
    return ((size_t)1 << (P::NB1 + k)) + (size_t)tile * P::SUBS * ((size_t)1 << k) + (size_t)(t - off);
}

// Bits of element j (0 .. 2^EB - 1) of a round placed at the plan's group positions.
template <int EB>
WG_HDC constexpr int round_bits(const RoundPlan& p, int j) {
    int r = 0;
    for (int k = 0; k < EB; ++k) r |= ((j >> k) & 1) << p.g[k];
    return r;
}

// Moduli for which the forward transform may skip the per-butterfly reduction of its upper
// input: each stage then adds at most 2q to a value's bound, so the at most 16 stages of
// N <= 2^16 take inputs below 4q to values below (4 + 2 x 16) q = 36 q < 2^64, and the Shoup
// lazy product accepts any 64-bit input.  The last phase then reduces the full word (reduce64)
// instead of a value below 4q.
constexpr uint64_t kLazyForwardLimit = uint64_t{1} << 58;
static_assert((4 + 2 * 16) < (1 << (64 - 58)), "lazy forward bound: 36 q < 2^64 for q < 2^58");

// The arithmetic of a round: the value a thread carries (as the word kept in shared memory), the
// butterflies of both directions, and the reductions a round needs at its stages' starts.
//
// WordArith: 64-bit words, Harvey / Shoup; LAZY (forward only, q < kLazyForwardLimit) keeps the
// upper value unreduced through the round.
template <bool LAZY>
struct WordArith {
    using V = uint64_t;
    uint64_t q;
    WG_HD static V of_bits(uint64_t x) { return x; }
    WG_HD static uint64_t bits(V v) { return v; }
    template <bool FWD, int EB, int RD>
    WG_HD void before_stage(V*, int) const {}
    WG_HD void forward(V& a, V& b, uint64_t w, uint64_t ws) const {
        const uint64_t two_q = q << 1;
        uint64_t t = a;
        if (!LAZY && t >= two_q) t -= two_q;
        const uint64_t u = mul_shoup_lazy(b, w, ws, q);
        a = t + u;
        b = t + two_q - u;
    }
    WG_HD void inverse(V& a, V& b, uint64_t w, uint64_t ws) const {
        const uint64_t two_q = q << 1;
        const uint64_t t = a, u = b;
        uint64_t sum = t + u;
        if (sum >= two_q) sum -= two_q;
        a = sum;
        b = mul_shoup_lazy(t - u + two_q, w, ws, q);
    }
};

// FpArith: signed integers in FP64 (wg_fp.cuh), q < fp::kLimit; the twiddle pair is (w, w / q).
// Bounds, in units of q, with values up to B q entering a product leaving at most 1/2 + B q 2^-55
// (at most 5/8 for B q <= 2^52):
//   forward, q < kNoReduce (2^42): each stage adds at most 5/8; inputs below 17 q (the base
//     changes of wg_ksfuse.cuh; 4 q elsewhere) stay below 17 + 16 x 5/8 = 27 q < 2^47.
//   forward, larger q (`red`): the rounds reduce to 1/2 every six (EB = 3) or four stages;
//     b -> b + 1/2 + b / 32 takes 1/2 to 3.85 in six stages, below the 4 q <= 2^52 a product takes.
//   inverse, q < kNoReduce: a sum doubles per stage; words below 4 q entering, and values reduced
//     to 1/2 between the two phases, stay below 4 x 2^8 q <= 2^52 through 8 stages.
//   inverse, larger q: values reduced to 1/2 at the start of a round and, for EB = 4, before its
//     third stage; at most three stages follow, and the sums stay below 4 q <= 2^52.
struct FpArith {
    using V = double;
    double q, inv_q;
    bool red;  // q >= kNoReduce
    WG_HD static V of_bits(uint64_t x) { return fp::bits_double(x); }
    WG_HD static uint64_t bits(V v) { return fp::double_bits(v); }
    template <bool FWD, int EB, int RD>
    WG_HD void before_stage(V* v, int s) const {
        const bool due = FWD ? (s == 0 && (EB == 4 || RD % 2 == 0)) : (s == 0 || (EB == 4 && s == 2));
        if (due && red) {
#pragma unroll
            for (int j = 0; j < (1 << EB); ++j) v[j] = fp::reduce(v[j], q, inv_q);
        }
    }
    WG_HD void forward(V& a, V& b, uint64_t w, uint64_t ws) const {
        const double t = a, u = fp::mulmod(b, fp::bits_double(w), fp::bits_double(ws), q);
        a = dadd(t, u);
        b = dadd(t, -u);
    }
    WG_HD void inverse(V& a, V& b, uint64_t w, uint64_t ws) const {
        const double t = a, u = b;
        a = dadd(t, u);
        b = fp::mulmod(dadd(t, -u), fp::bits_double(w), fp::bits_double(ws), q);
    }
};
WG_HD FpArith fp_arith(const Modulus& m) { return FpArith{m.qd, m.inv_q, m.q >= fp::kNoReduce}; }

// Thread (sub, o)'s elements in round RD: base | round_bits(j) within its sub-transform, with base's
// bits disjoint from the group positions, so every index splits into a runtime part (one per round,
// or one per stage for twiddles) plus a compile-time offset: pad16, shifts and the tile's offsets
// distribute over disjoint bit sets.  Accesses then use immediate offsets, and butterflies of a
// stage that share a twiddle load it once (same address).
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int RD, int TL = kMaxTile>
struct Round {
    using P = Phase<LOGN, FWD, COLS, EB, STAGED, TL>;
    static constexpr int E = P::E;
    // the elements of a thread are consecutive words of the limb
    static constexpr bool RUN = !COLS && make_plan<P::MB, FWD, EB>(RD).g[EB - 1] == EB - 1;
    WG_HD static int base(int o) {
        constexpr RoundPlan plan = make_plan<P::MB, FWD, EB>(RD);
#pragma unroll
        for (int k = 0; k < EB; ++k) o = insert_zero(o, plan.g[k]);
        return o;
    }
    WG_HD static int element(int sub, int o) { return COLS ? base(o) * P::SUBS + sub : (sub << P::MB) | base(o); }
    // offsets of element j from element(): in the tile, and in the limb
    WG_HDC static constexpr int tile_step(int j) {
        return round_bits<EB>(make_plan<P::MB, FWD, EB>(RD), j) * (COLS ? P::SUBS : 1);
    }
    WG_HDC static constexpr size_t limb_step(int j) {
        return (size_t)round_bits<EB>(make_plan<P::MB, FWD, EB>(RD), j) << (COLS ? P::NB2 : 0);
    }
    template <class Arith>
    WG_HD static void scatter(uint64_t* sm, int sub, int o, const typename Arith::V* v) {
        uint64_t* row = sm + pad16(element(sub, o));
#pragma unroll
        for (int j = 0; j < E; ++j) row[pad16(tile_step(j))] = Arith::bits(v[j]);
    }
    template <class Arith>
    WG_HD static void gather(const uint64_t* sm, int sub, int o, typename Arith::V* v) {
        const uint64_t* row = sm + pad16(element(sub, o));
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = Arith::of_bits(row[pad16(tile_step(j))]);
    }
    // The round's stages (up to EB radix-2 stages) on the thread's elements.  `tw` is the CTA's
    // staged block (STAGED, twiddle_src order) or the modulus's table of this direction.
    template <class Arith>
    WG_HD static void stages(typename Arith::V* v, int sub, int o, int tile, const Arith& ar,
                             const TwPair* __restrict__ tw) {
        constexpr RoundPlan plan = make_plan<P::MB, FWD, EB>(RD);
        const int b0 = base(o);
#pragma unroll
        for (int s = 0; s < plan.ns; ++s) {
            ar.template before_stage<FWD, EB, RD>(v, s);
            const int b = plan.sb[s];
            const int jb = plan.jb[s];
            // The table index of a pair is (1 << (n-1-gb)) + (x >> (gb+1)) for its global index x
            // and stage bit gb; relative to the staged block (or to the table) it is:
            const int kr = P::NB2 - 1 - b;  // row-stage of bit b
            const size_t base_idx =
                COLS ? (size_t)(1 << (P::NB1 - 1 - b))
                     : (STAGED ? (size_t)(P::SUBS * ((1 << kr) - 1) + (sub << kr))
                               : ((size_t)1 << (P::NB1 + kr)) + (size_t)tile * P::SUBS * ((size_t)1 << kr) +
                                     (size_t)(sub << kr));
            // (in the round of the lowest bits the table is in row_order: thread-minor)
            const TwPair* tw_st = tw + base_idx + (RUN ? o : b0 >> (b + 1));
#pragma unroll
            for (int j = 0; j < E; ++j) {
                if ((j >> jb) & 1) continue;
                const int j1 = j | (1 << jb);
                const int k = (round_bits<EB>(plan, j) >> (b + 1)) << (RUN ? P::OB : 0);
#if defined(__CUDA_ARCH__)
                uint64_t w, ws;
                if (STAGED) {
                    const TwPair tp = tw_st[k];
                    w = tp.w;
                    ws = tp.ws;
                } else {
                    const ulonglong2 tp = __ldg(reinterpret_cast<const ulonglong2*>(tw_st + k));
                    w = tp.x;
                    ws = tp.y;
                }
#else
                const uint64_t w = tw_st[k].w, ws = tw_st[k].ws;
#endif
                if (FWD)
                    ar.forward(v[j], v[j1], w, ws);
                else
                    ar.inverse(v[j], v[j1], w, ws);
            }
        }
    }
};

// Words of an FP64 transform on their way in and out of a phase.  Between the two phases (and the
// fused kernels' steps) a limb holds the bits of the doubles; the inverse transform's first phase
// reduces them there when its rounds do not (q < kNoReduce).
WG_HD uint64_t fp_load(bool first, uint64_t x, const Modulus& m) {
    if (!first) return x;
    if (x >> 52) x = reduce64(x, m);  // words of 4 q and more, which the forward transform accepts
    return fp::double_bits(fp::from_word(x));
}
WG_HD uint64_t fp_store(bool last, bool fwd, uint64_t x, const Modulus& m) {
    const double v = fp::bits_double(x);
    if (!last) return !fwd && m.q < fp::kNoReduce ? fp::double_bits(fp::reduce(v, m.qd, m.inv_q)) : x;
    if (fwd) return fp::canonical(v, m.qd, m.inv_q);
    return fp::to_word(fp::lift(fp::mulmod(v, m.n_inv_w, m.n_inv_wq, m.qd), m.qd));
}

// The forward row phase of one limb (data: after the forward column phase, read only) with an
// element-wise epilogue on the finished canonical words v instead of storing them:
//   kEpiRescale: out = (in - v) * p^-1 mod q  (in reduced below q first; c0, c1 = p^-1 and its
//                Shoup constant: the rescale finish step, as kb_rescale_finish);
//   kEpiCombine: out = c0 ? in + (acc - v) : acc - v  (the key switch's final combine, as
//                combine_coeff).
// out may alias in or acc (each word is read and written by the same thread).
enum NttEpilogue : int { kEpiRescale = 1, kEpiCombine = 2 };
struct NttEpiJob {
    const uint64_t* data;
    const uint64_t* acc;
    const uint64_t* in;
    uint64_t* out;
    uint64_t c0, c1;
    int mod;
    int kind;
};

// The epilogue's word for the finished canonical word v and the operands acc, in (each used
// only where the kind needs it).
WG_HD uint64_t epilogue_value(const NttEpiJob& j, uint64_t acc, uint64_t in, uint64_t v, uint64_t q) {
    if (j.kind == kEpiRescale) {
        if (in >= q) in -= q;
        return mul_shoup(sub_mod(in, v, q), j.c0, j.c1, q);
    }
    const uint64_t d = sub_mod(acc, v, q);
    return j.c0 ? add_mod(in, d, q) : d;
}

// The epilogue at word off of the job's limbs, operands read from their arrays.
WG_HD void ntt_epilogue(const NttEpiJob& j, size_t off, uint64_t v, uint64_t q) {
    const uint64_t acc = j.kind == kEpiCombine ? j.acc[off] : 0;
    const uint64_t in = (j.kind == kEpiRescale || j.c0) ? j.in[off] : 0;
    j.out[off] = epilogue_value(j, acc, in, v, q);
}

// Words of a word-arithmetic limb on their way out of its last phase.
WG_HD uint64_t word_store(bool last, bool fwd, uint64_t v, const Modulus& m) {
    if (!last) return v;
    if (!fwd) return mul_shoup(v, m.n_inv, m.n_inv_shoup, m.q);
    return m.q < kLazyForwardLimit ? reduce64(v, m) : red4q(v, m.q);
}

// Key products on 8 coefficients of a thread, between the rounds of k_rows_mac (wg_ntt.cu): `own` and
// `digit` take a key-term word and a digit's word before its row phase, `transformed` what its rounds
// leave, `add` the products with the key words of one of the two polynomials; `value` is the sum as
// the inverse row phase starts from it and `row_word` a word that phase ends with, `words` the
// canonical sum.
// FP64: |transformed word| <= 27 q where the modulus needs no reduction (FpArith), so its product with a
// key word (key_factor) has |a wq| < 2^47.
struct MacSumsFp {
    using V = double;
    double s[2][8];
    WG_HD void clear() {
#pragma unroll
        for (int k = 0; k < 8; ++k) s[0][k] = s[1][k] = 0.0;
    }
    WG_HD static V own(uint64_t w) { return fp::from_word(w); }
    WG_HD static V digit(uint64_t w) { return fp::bits_double(w); }
    WG_HD static void transformed(V* v, const Modulus& m) {
        if (m.q < fp::kNoReduce) return;
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = fp::reduce(v[k], m.qd, m.inv_q);
    }
    WG_HD void add(int poly, const V* v, const uint64_t* key, int part, const Modulus& m) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const fp::Factor f = fp::key_factor(key[k], m.inv_q);
            s[poly][k] = fp::mont_sum_bound(dadd(s[poly][k], fp::mulmod(v[k], f.w, f.wq, m.qd)), part, m);
        }
    }
    WG_HD V value(int poly, int k, const Modulus& m) const { return fp::mont_sum_value(s[poly][k], m); }
    WG_HD static uint64_t row_word(V v, const Modulus& m) { return fp_store(false, false, fp::double_bits(v), m); }
    WG_HD uint64_t word(int poly, int k, const Modulus& m) const { return fp::mont_sum_word(s[poly][k], m); }
};
// The same in words.
struct MacSumsWords {
    using V = uint64_t;
    WideSum s[2][8];
    WG_HD void clear() {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            s[0][k].clear();
            s[1][k].clear();
        }
    }
    WG_HD static V own(uint64_t w) { return w; }
    WG_HD static V digit(uint64_t w) { return w; }
    WG_HD static void transformed(V* v, const Modulus& m) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = word_store(true, true, v[k], m);
    }
    WG_HD void add(int poly, const V* v, const uint64_t* key, int, const Modulus& m) {
#pragma unroll
        for (int k = 0; k < 8; ++k) s[poly][k].add(v[k], key[k], m);
    }
    WG_HD V value(int poly, int k, const Modulus& m) const { return s[poly][k].mont_value(m); }
    WG_HD static uint64_t row_word(V v, const Modulus&) { return v; }
    WG_HD uint64_t word(int poly, int k, const Modulus& m) const { return s[poly][k].mont_value(m); }
};

// Global offset (within one limb) of tile element e.
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL = kMaxTile>
WG_HD size_t tile_offset(int tile, int e) {
    using P = Phase<LOGN, FWD, COLS, EB, STAGED, TL>;
    if (COLS) {
        const int hh = e / P::SUBS, c = e % P::SUBS;
        return ((size_t)hh << P::NB2) + (size_t)tile * P::SUBS + c;
    }
    return (size_t)tile * P::TILE + e;
}

// The epilogue of an FP64 transform: v is the unreduced value of the last row phase's word.  The
// rescale's product runs in FP64 as well; the combine keeps the word arithmetic, because `in` may
// hold a word in [q, 2q) (a product with a single Barrett correction) that add_mod carries on.
struct FpEpilogue {
    double w, wq;
};
WG_HD FpEpilogue fp_epilogue(const NttEpiJob& j, const Modulus& m) {
    FpEpilogue c{0.0, 0.0};
    if (j.kind == kEpiRescale) fp::factor_of(j.c0, m.qd, m.inv_q, c.w, c.wq);
    return c;
}
WG_HD uint64_t fp_epilogue_value(const NttEpiJob& j, const FpEpilogue& c, uint64_t acc, uint64_t in, uint64_t x,
                                 const Modulus& m) {
    const double v = fp::reduce(fp::bits_double(x), m.qd, m.inv_q);
    if (j.kind == kEpiRescale) {
        // |in - v| <= 2^51 + q / 2 (any larger word is reduced first): the product stays below q in
        // magnitude (1/2 + |in - v| 2^-53, factor_of)
        if (in >> 51) in = reduce64(in, m);
        const double d = dadd(fp::from_word(in), -v);
        return fp::to_word(fp::lift(fp::mulmod(d, c.w, c.wq, m.qd), m.qd));
    }
    return epilogue_value(j, acc, in, fp::to_word(fp::lift(v, m.qd)), m.q);
}

// A whole transform in one launch: the limb's TL-element tiles of both phases belong to the CTAs of
// one cluster, which hand the first phase's results to the second through distributed shared memory.
// Tile element e of the first phase goes to element `at` of CTA `cta`'s second-phase tile.
constexpr int kWholeMaxLog = 14;
template <int LOGN>
struct Whole {
    static_assert(LOGN <= kWholeMaxLog, "a cluster has at most 8 CTAs");
    static constexpr int N = 1 << LOGN;
    static constexpr int TL = N < kMaxTile ? N : kMaxTile;
    static constexpr int CTAS = N / TL;  // the cluster: 1 to 8 CTAs
    template <bool FWD, bool COLS>
    using Ph = Phase<LOGN, FWD, COLS, 3, false, TL>;
    static constexpr int COLUMNS = Ph<true, true>::SUBS;  // columns, and rows, of a CTA's tiles
    static constexpr int ROWS = Ph<true, false>::SUBS;
    static constexpr int NB2 = Ph<true, true>::NB2;
    static constexpr int PAD = TL + TL / 16;
};
struct HandOver {
    int cta, at;
};
template <int LOGN, bool FWD>
WG_HD HandOver hand_over(int tile, int e) {
    using W = Whole<LOGN>;
    if (FWD) {  // columns to rows
        const int h = e / W::COLUMNS, c = tile * W::COLUMNS + e % W::COLUMNS;
        return {h / W::ROWS, (h % W::ROWS) << W::NB2 | c};
    }
    const int h = tile * W::ROWS + (e >> W::NB2), c = e & ((1 << W::NB2) - 1);
    return {c / W::COLUMNS, h * W::COLUMNS + c % W::COLUMNS};
}

// Whether `transforms` limbs of a ring go in one launch each way (Whole) or in two phases: one launch for
// the rings whose limb a cluster of small CTAs covers, while the batch is about one wave of clusters.
// Forward at 38-bit moduli, one launch / two phases, as calls one after the other, in us: 2^14: 8 / 12 (12
// limbs), 10 / 12 (32), 14 / 17 (64); 2^13: 9 / 12 (64), 12 / 14 (128), 21 / 21 (256).  Device time alone:
// 2^14: 5.6 / 6.2 (12), 7.7 / 6.3 (16), 7.9 / 8.4 (24), 12.8 / 13.0 (64), 20.5 / 20.5 (128); 2^13: 7.3 / 7.9 (64);
// 2^12: 6.4 / 7.5 (128), 54 / 59 (2048); 2^10: 3.2 / 4.4 (64), 12.8 / 17.2 (2048).  At 60 bits: 2^14: 7.3 / 7.7 (12),
// 10.7 / 7.8 (16), 10.8 / 11.4 (24), 14.5 / 15.0 (48), 19.0 / 18.3 (64); 2^13: 17.0 / 17.3 (128); 2^12: 90.7 / 90.8 (2048);
// 2^10: 20.5 / 22.8 (2048).  So chains with word moduli stop at 48 limbs of 2^14 and leave out the launches
// that fit one CTA an SM where the clusters of 8 do not (13 to 18 limbs; with 38 bits there the call with
// one launch is still the shorter one, 10 / 12).  At 2^15 clusters of 8 CTAs of 512 threads leave most
// SMs waiting (29 / 24 at 64 limbs, 189 / 132 at 512), so larger rings take the phases.
inline bool whole_launch(int logN, size_t transforms, int sm_count, bool word_moduli) {
    if (logN <= 12) return true;
    if (logN > kWholeMaxLog || transforms << logN > (size_t{1} << 20)) return false;
    if (logN < kWholeMaxLog || !word_moduli) return true;
    const size_t ctas = (transforms << logN) / kMaxTile;
    return transforms <= 12 || (ctas > (size_t)sm_count && transforms <= 48);
}

// The geometry (kNttGeometries order) of one phase over `words` residues where `tuned` is the best of
// large batches: in small launches 8 residues a thread in place of 16, which halve the threads.
// Device time with 8 and 16 in us: forward row phases of 60-bit moduli at 2^15, 4 limbs 7.9 and 8.8, 8
// limbs 8.0 and 9.3, 24 limbs 15.7 and 16.2, 32 limbs 19.3 and 19.1; inverse ones of 38-bit moduli, 8
// limbs 6.4 and 6.8, 17 limbs 8.3 and 8.8, 34 limbs 12.6 and 12.8, 68 limbs 21.3 and 21.2; inverse column
// phases of the walsh15 chain, 13 limbs 9.4 and 9.8, 26 limbs 11.6 and 11.6, 52 limbs 19.3 and 18.2.
inline int launch_geometry(int tuned, bool cols, size_t words, int sm_count, bool word_moduli) {
    const size_t small = (size_t)sm_count * kMaxTile * (word_moduli && !cols ? 3 : 2);
    return tuned >= 2 && words <= small ? tuned - 2 : tuned;
}

// The place of twiddle x of a row (of the 2^kr of row-stage kr = NB2 - 1 - b) in the table.  In the
// round of a row's lowest bits thread o uses the 2^(eb-1-b) consecutive twiddles from o << (eb-1-b),
// so over a warp each of these loads would touch a 128-byte line per lane; there they stand
// thread-minor.
WG_HD size_t row_order(int nb2, int eb, int b, size_t x) {
    const int last = nb2 - eb * ((nb2 + eb - 1) / eb - 1);  // stages of that round
    if (b >= last) return x;
    const int kb = eb - 1 - b, ob = nb2 - eb;
    return ((x & (((size_t)1 << kb) - 1)) << ob) | (x >> kb);
}

// The place of twiddle i of a ring of 2^n in the table of the geometries of 2^eb residues per thread: rows
// in row_order.
WG_HD size_t twiddle_place(int n, int eb, size_t i) {
    const int nb1 = n / 2, nb2 = n - nb1;
    if (i < ((size_t)1 << nb1)) return i;
    const int kr = floor_log2((unsigned)i) - nb1;
    const size_t stage = (size_t)1 << (nb1 + kr), row = (i - stage) >> kr, x = i & (((size_t)1 << kr) - 1);
    return stage + (row << kr) + row_order(nb2, eb, nb2 - 1 - kr, x);
}

// An entry of a modulus's table from its split (w, Shoup w) words: the factor pair (w, w / q) as bits of
// doubles for the moduli of the FP64 path (unless `words`), the words otherwise.
WG_HD TwPair twiddle_pair(uint64_t w, uint64_t ws, uint64_t q, bool words) {
    if (q >= fp::kLimit || words) return TwPair{w, ws};
    double f, fq;
    fp::factor(w, q, f, fq);
    return TwPair{fp::double_bits(f), fp::double_bits(fq)};
}

}  // namespace ntt
}  // namespace wg
