// Per-thread steps of the fused key-switch and rescale kernels (wg_ksfuse.cu), shared with the CPU
// emulation test, which runs them thread by thread between the same barriers.
//
// The fused kernels work on one column tile of the two-phase NTT (wg_ntt.cu): the TILE
// coefficients {(h << NB2) + tile * SUBS + c : h < 2^NB1, c < SUBS}, i.e. SUBS whole columns.
// The inverse transform ends with the column phase and the forward transform starts with it,
// and both phases cover exactly these coefficients, so a CTA can finish the inverse transform
// of some limbs, combine them coefficient by coefficient, and start the forward transform of
// the results without a pass through device memory in between:
//
//   ModUp:   inverse column phase of the digit's alpha source limbs (their row phase ran as one
//            batched launch), N^-1 scaling, the HPS base change of modup_coeff_w
//            (wg_keyswitch.cuh; apply_hps_crt_base_change, ckks_keyswitch.cpp:278-332), then the
//            forward column phase of every destination limb;
//   ModDown: inverse column phase of the K P limbs of one accumulator, N^-1 scaling, the folded
//            ModDown of moddown_all_limbs (ckks_apply_folded_approx_crt_moddown_pair_eval_q,
//            ckks_keyswitch.cpp:521-607), then the forward column phase of every Q limb;
//   Rescale: inverse column phase of the dropped limb, N^-1 scaling, the rounded remainder
//            for every lower limb, then the forward column phase of each remainder (the row
//            phase that follows finishes the rescale in its epilogue, k_ntt_rows_epi).
//
// The butterflies, reductions and FP64 sums are those of the unfused kernels in the same
// order, so the words written equal the ones the separate launches write.
//
// A thread owns the same elements of the tile in the inverse phase's last round as in the forward
// phase's first (make_plan), so between the two transforms everything is its own: the finished
// source limbs wait in shared memory slots that only their thread touches (slot k * THREADS + t: no
// barrier, no bank conflict, no padding), and a base change's values go from registers straight
// into the forward rounds.  Only the rounds' exchanges use the padded tile and barriers.
//
// Limbs whose modulus is below fp::kLimit run in FP64 (wg_fp.cuh): their slots hold doubles, from
// the inverse row phase's words to those the forward row phase continues from.  A scaled source
// (ModUp), P residue (ModDown) or dropped limb (rescale) is then the same canonical residue as
// its word, as a double (SourceKinds, fp_src: a bit per source limb for the form its slots hold).
#pragma once
#include <cstddef>
#include <cstdint>

#include "wg_keyswitch.cuh"
#include "wg_ntt.cuh"

namespace wg {
namespace ksf {

// Column tile of the fused kernels: 1024 elements, so the source tiles of a digit or of the P limbs fit
// in shared memory several CTAs per SM.
constexpr int kTile = 1024;

// EB: a thread carries 2^EB residues, 8 or 4 (128 or 256 threads a tile).  Four hold 64 registers, so the
// same tiles keep twice the warps on an SM, at one round's exchange more and half the sums per table
// entry read: measured (us) against eight, the ModUp of a Walsh AES takes 97400 against 105000, its
// ModDown 120500 against 122700, and in one bootstrap 1140 against 1273 and 1070 against 1171 (61-bit
// words: long serial chains of integer products); on the all-FP64 XBOOT chain the ModUp of a bootstrap
// takes 5510 against 4910 but the ModDown 3205 against 3434, and a rescale is 2 to 10 % slower.
constexpr int kModUpBits = 2;    // chains with word moduli (from fp::kLimit up)
constexpr int kModUpFpBits = 3;  // chains without
constexpr int kModDownBits = 2;
constexpr int kRescaleBits = 3;

template <int LOGN, int EB>
struct Geom {
    using Fwd = ntt::Phase<LOGN, true, true, EB, false, kTile>;
    using Inv = ntt::Phase<LOGN, false, true, EB, false, kTile>;
    template <int RD>
    using FwdRound = ntt::Round<LOGN, true, true, EB, false, RD, kTile>;
    template <int RD>
    using InvRound = ntt::Round<LOGN, false, true, EB, false, RD, kTile>;
    static constexpr int LOG = LOGN, BITS = EB;
    static constexpr int N = 1 << LOGN;
    static constexpr int TILE = Fwd::TILE;
    static constexpr int THREADS = Fwd::THREADS;
    static constexpr int E = 1 << EB;
    static constexpr int PAD = TILE + TILE / 16;  // words of the padded exchange tile
    static constexpr int TILES = N / TILE;
    static constexpr int ROUNDS = Fwd::ROUNDS;
    static_assert(Fwd::TILE == Inv::TILE && Fwd::THREADS == Inv::THREADS, "one tile shape for both directions");
};

// The column tile of block `x` of a job's `blocks` = TILES * split and the outputs begin, begin + step, ...
// it makes.  (Every step-th and not a run, so that the word moduli, which cost several times an FP64
// one and stand together at the end, spread over the blocks.)
struct Share {
    int tile, begin, step;
};
WG_HD Share share_of(unsigned x, unsigned blocks, unsigned tiles) {
    return {(int)(x % tiles), (int)(x / tiles), (int)(blocks / tiles)};
}

// Offset in the limb of thread t's element 0 in a round; element k is limb_step(k) further.
template <class R>
WG_HD size_t limb_offset(int tile, int t) {
    using P = typename R::P;
    const int e = R::element(P::sub_of(t), P::o_of(t));
    return ((size_t)(e / P::SUBS) << P::NB2) + (size_t)tile * P::SUBS + e % P::SUBS;
}

#if defined(__CUDACC__)
// Thread t's elements (first inverse round) of one limb into its slots, as asynchronous copies
// (cp.async, 8 bytes each) that pass no register, so a CTA can have all its source limbs in flight at
// once; completion is awaited per commit group (cp_async_wait_upto), by the thread alone.
template <class G>
__device__ __forceinline__ void load_slots_async(uint64_t* slots, const uint64_t* __restrict__ limb, int tile, int t) {
    using R = typename G::template InvRound<0>;
    const uint64_t* p = limb + limb_offset<R>(tile, t);
#pragma unroll
    for (int k = 0; k < G::E; ++k) {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(slots + k * G::THREADS + t);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(p + R::limb_step(k)) : "memory");
    }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int P>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(P) : "memory");
}
// wait until at most `pending` of this thread's commit groups are still in flight
__device__ __forceinline__ void cp_async_wait_upto(int pending) {
    switch (pending) {
        case 0: cp_async_wait<0>(); break;
        case 1: cp_async_wait<1>(); break;
        case 2: cp_async_wait<2>(); break;
        case 3: cp_async_wait<3>(); break;
        case 4: cp_async_wait<4>(); break;
        case 5: cp_async_wait<5>(); break;
        case 6: cp_async_wait<6>(); break;
        default: cp_async_wait<7>(); break;
    }
}
#endif

// Thread t's elements of a limb's tile in round R, and back (no reduction: the forward transform's
// row phase continues from these words).
template <class R>
WG_HD void load_limb(uint64_t* w, const uint64_t* __restrict__ limb, int tile, int t) {
    const uint64_t* p = limb + limb_offset<R>(tile, t);
#pragma unroll
    for (int k = 0; k < R::E; ++k) w[k] = p[R::limb_step(k)];
}
template <class R>
WG_HD void store_limb(const uint64_t* w, uint64_t* __restrict__ limb, int tile, int t) {
    uint64_t* p = limb + limb_offset<R>(tile, t);
#pragma unroll
    for (int k = 0; k < R::E; ++k) p[R::limb_step(k)] = w[k];
}

// Per source limb (bits): its slots hold doubles; its modulus is of the FP64 path but not below
// fp::kNoReduce.
struct SourceKinds {
    unsigned fp64 = 0, wide = 0;
    WG_HD void set(int i, uint64_t q) {
        if (q < fp::kLimit) fp64 |= 1u << i;
        if (q < fp::kLimit && q >= fp::kNoReduce) wide |= 1u << i;
    }
};

// A slot's word as an integer, whichever form it holds.
WG_HD uint64_t slot_word(uint64_t x, bool fp64) { return fp64 ? fp::to_word(fp::bits_double(x)) : x; }

// Last step of an FP64 inverse transform: multiply by the factor pair (N^-1, or N^-1 with a base
// change's constant) to the canonical residue.
template <int E>
WG_HD void scale_fp(double* v, double w, double wq, double q) {
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = fp::lift(fp::mulmod(v[k], w, wq, q), q);
}

// Last step of the inverse transform: multiply by N^-1 (canonical).
template <int E>
WG_HD void scale_n_inv(uint64_t* v, const Modulus& m) {
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = mul_shoup(v[k], m.n_inv, m.n_inv_shoup, m.q);
}

// ModUp, source limb i of the digit (canonical coefficients): scale by qhat_inv_i in place and add
// the FP64 estimate term to the alpha sums, in the order of modup_coeff_w.  (modup_coeff_w first
// reduces its input below q; the inverse transform's N^-1 step already leaves it canonical, so that
// reduction is the identity here.)
template <class G, class Desc>
WG_HD void modup_scale(uint64_t* v, const Desc& d, int i, uint64_t qi, double* alpha) {
    const uint64_t w = WG_LDG(d.qhat_inv + i), ws = WG_LDG(d.qhat_inv_s + i);
    const double inv = WG_LDG(d.src_inv + i);
#pragma unroll
    for (int k = 0; k < G::E; ++k) {
        v[k] = mul_shoup(v[k], w, ws, qi);
        alpha[k] = dadd(alpha[k], dmul(u2d(v[k]), inv));
    }
}

// The same for an FP64 source, from the inverse rounds' values: N^-1 and qhat_inv_i in one factor.
template <class G, class Desc>
WG_HD void modup_scale_fp(double* v, const Desc& d, int i, double qi, double* alpha) {
    const ntt::TwPair f = d.scale_fp[i];
    scale_fp<G::E>(v, fp::bits_double(f.w), fp::bits_double(f.ws), qi);
    const double inv = WG_LDG(d.src_inv + i);
#pragma unroll
    for (int k = 0; k < G::E; ++k) alpha[k] = dadd(alpha[k], dmul(v[k], inv));
}

WG_HD uint32_t hps_count(double alpha, int n) {
    uint64_t h = round_half_up(alpha);
    return (uint32_t)(h > (uint64_t)n ? (uint64_t)n : h);
}

// ModUp destination dst of the digit: thread t's coefficients.
// src holds the n scaled sources' slots (TILE words each).
template <class G, class Desc>
WG_HD void modup_value(uint64_t* v, const uint64_t* src, int t, const Desc& d, int dst, uint64_t m, const uint32_t* hps,
                       unsigned fp_src) {
    const int n = d.src_count;
    const uint64_t* row = d.qhat + (size_t)dst * n;
    const uint64_t* row_s = d.qhat_s + (size_t)dst * n;
    const uint64_t* corr = d.corr + (size_t)dst * (n + 1);
#pragma unroll
    for (int k = 0; k < G::E; ++k) v[k] = 0;
    for (int i = 0; i < n; ++i) {
        const uint64_t w = WG_LDG(row + i), ws = WG_LDG(row_s + i);
#pragma unroll
        for (int k = 0; k < G::E; ++k)
            v[k] = add_mod(v[k], mul_shoup(slot_word(src[i * G::TILE + k * G::THREADS + t], fp_src >> i & 1), w, ws, m), m);
    }
#pragma unroll
    for (int k = 0; k < G::E; ++k) v[k] = sub_mod(v[k], WG_LDG(corr + hps[k]), m);
}

// Sums of products s w of thread t's source elements s, modulo a destination q of the FP64 path.
//   q < fp::kNoReduce: exact sums with one reduction (fp::Dot), 4 FP64 instructions a term; a word
//     source (61 bits) is two terms, s = s1 2^31 + s0 with the factors w and 2^31 w; a 43- to 50-bit
//     FP64 source would overflow the sum and adds its reduced product instead.
//   larger q: an FP64 source adds the reduced product through its factor pair (w, w / q), a word
//     source a lazy Shoup product in [0, 2q), centred; each term adds at most q in magnitude, and the
//     sum is brought back to q / 2 after every fourth, so it stays below 5.5 q < 2^53.
// `f` is the term's table entry: (w, w / q), or (w, 2^31 w) for a word source (fp::kWordSplit).
template <class G>
struct SumFp {
    fp::Dot d[G::E];
    WG_HD void start(int k, double v) {
        d[k].clear();
        d[k].l = v;
    }
    WG_HD void add(const uint64_t* slots, int t, bool fp64, bool wide, ntt::TwPair f, uint64_t w, uint64_t ws, int term,
                   const Modulus& m) {
        const double f0 = fp::bits_double(f.w), f1 = fp::bits_double(f.ws);
        const bool dot = m.q < fp::kNoReduce;
        slots += t;
        if (fp64 && dot && !wide) {
#pragma unroll
            for (int k = 0; k < G::E; ++k) d[k].add(fp::bits_double(slots[k * G::THREADS]), f0);
        } else if (fp64) {
#pragma unroll
            for (int k = 0; k < G::E; ++k)
                d[k].l = dadd(d[k].l, fp::mulmod(fp::bits_double(slots[k * G::THREADS]), f0, f1, m.qd));
        } else if (dot) {
#pragma unroll
            for (int k = 0; k < G::E; ++k) {
                const uint64_t s = slots[k * G::THREADS];
                d[k].add(fp::from_word(s & 0x7fffffffu), f0);
                d[k].add(fp::from_word(s >> 31), f1);
            }
        } else {
#pragma unroll
            for (int k = 0; k < G::E; ++k) {
                const uint64_t r = mul_shoup_lazy(slots[k * G::THREADS], w, ws, m.q);
                d[k].l = dadd(d[k].l, dadd(fp::from_word(r), -m.qd));
            }
        }
        if (!dot && (term & 3) == 3) {
#pragma unroll
            for (int k = 0; k < G::E; ++k) d[k].l = fp::reduce(d[k].l, m.qd, m.inv_q);
        }
    }
    WG_HD void finish(double* v, const Modulus& m) const {
        const bool dot = m.q < fp::kNoReduce;
#pragma unroll
        for (int k = 0; k < G::E; ++k) v[k] = dot ? d[k].value(m.qd, m.inv_q) : d[k].l;
    }
};
static_assert(2 * kMaxDigitWidth <= fp::kDotTerms && 2 * kMaxPLimbs <= fp::kDotTerms, "a base change is one exact sum");

// ModUp destination dst of the FP64 path: thread t's coefficients, unreduced.
template <class G, class Desc>
WG_HD void modup_value_fp(double* v, const uint64_t* src, int t, const Desc& d, int dst, const Modulus& m,
                          const uint32_t* hps, SourceKinds kinds) {
    const int n = d.src_count;
    const uint64_t* corr = d.corr + (size_t)dst * (n + 1);
    SumFp<G> sum;
#pragma unroll
    for (int k = 0; k < G::E; ++k) sum.start(k, -fp::from_word(WG_LDG(corr + hps[k])));
    for (int i = 0; i < n; ++i) {
        const size_t at = (size_t)dst * n + i;
        sum.add(src + i * G::TILE, t, kinds.fp64 >> i & 1, kinds.wide >> i & 1, d.qhat_fp[at], d.qhat[at], d.qhat_s[at], i,
                m);
    }
    sum.finish(v, m);
}

// ModDown: FP64 estimate of thread t's coefficients over the K P limbs, in the order of
// moddown_all_limbs_k; FMA: rounded as a fused multiply-add (the pair ModDown's compiled form)
// or as a multiply then an add (the single-polynomial ModDown's).  The slots hold canonical
// residues (the inverse transform's N^-1 step), so moddown_all_limbs_k's reduction of its input
// below p is the identity here and is left out.
template <class G, bool FMA = true>
WG_HD void moddown_hps(const uint64_t* src, int t, const Modulus* __restrict__ pmods, int K, uint32_t* hps,
                       unsigned fp_src) {
    double alpha[G::E];
#pragma unroll
    for (int k = 0; k < G::E; ++k) alpha[k] = 0.0;
    for (int pi = 0; pi < K; ++pi) {
        const double inv = pmods[pi].inv_q;
#pragma unroll
        for (int k = 0; k < G::E; ++k) {
            const uint64_t x = src[pi * G::TILE + k * G::THREADS + t];
            const double s = fp_src >> pi & 1 ? fp::bits_double(x) : u2d(x);
            alpha[k] = FMA ? dfma(s, inv, alpha[k]) : dadd(alpha[k], dmul(s, inv));
        }
    }
#pragma unroll
    for (int k = 0; k < G::E; ++k) hps[k] = hps_count(alpha[k], K);
}

// ModDown contribution for Q limb qi: thread t's coefficients (canonical P residues as for
// moddown_hps).
template <class G>
WG_HD void moddown_value(uint64_t* v, const uint64_t* src, int t, int K, uint64_t q, const uint64_t* __restrict__ iv,
                         const uint64_t* __restrict__ ivs, const uint32_t* hps, unsigned fp_src) {
#pragma unroll
    for (int k = 0; k < G::E; ++k) v[k] = 0;
    for (int pi = 0; pi < K; ++pi) {
        const uint64_t w = WG_LDG(iv + pi), ws = WG_LDG(ivs + pi);
#pragma unroll
        for (int k = 0; k < G::E; ++k)
            v[k] = add_mod(v[k], mul_shoup(slot_word(src[pi * G::TILE + k * G::THREADS + t], fp_src >> pi & 1), w, ws, q), q);
    }
#pragma unroll
    for (int k = 0; k < G::E; ++k) v[k] = sub_mod(v[k], (uint64_t)hps[k], q);
}

// The same for a Q limb of the FP64 path, unreduced.
template <class G>
WG_HD void moddown_value_fp(double* v, const uint64_t* src, int t, int K, const Modulus& m,
                            const uint64_t* __restrict__ iv, const uint64_t* __restrict__ ivs,
                            const ntt::TwPair* __restrict__ ivf, const uint32_t* hps, SourceKinds kinds) {
    SumFp<G> sum;
#pragma unroll
    for (int k = 0; k < G::E; ++k) sum.start(k, -fp::from_word(hps[k]));
    for (int pi = 0; pi < K; ++pi)
        sum.add(src + pi * G::TILE, t, kinds.fp64 >> pi & 1, kinds.wide >> pi & 1, ivf[pi], iv[pi], ivs[pi], pi, m);
    sum.finish(v, m);
}

// Rescale: thread t's rounded remainders of the dropped limb (slots, canonical, modulus p) for
// target limb q, as kb_rescale_prep forms them
// (ckks_rescale, src/ckks/operations/arith/ckks_rescale.cpp:68-148).
template <class G>
WG_HD void rescale_value(uint64_t* v, const uint64_t* drop, int t, uint64_t p, uint64_t q, uint64_t one_s, uint64_t half,
                         bool fp_drop) {
#pragma unroll
    for (int k = 0; k < G::E; ++k) {
        uint64_t shift = slot_word(drop[k * G::THREADS + t], fp_drop) + (p >> 1);
        if (shift >= p) shift -= p;
        v[k] = sub_mod(reduce_shoup(shift, q, one_s), half, q);
    }
}

// The same for a target limb of the FP64 path: unreduced, at most 2 q in magnitude.
template <class G>
WG_HD void rescale_value_fp(double* v, const uint64_t* drop, int t, uint64_t p, const Modulus& m, uint64_t one_s,
                            uint64_t half, bool fp_drop) {
    const double h = fp::from_word(half);
    const double pd = u2d(p), hp = u2d(p >> 1);
#pragma unroll
    for (int k = 0; k < G::E; ++k) {
        const uint64_t x = drop[k * G::THREADS + t];
        double r;
        if (fp_drop) {
            double shift = dadd(fp::bits_double(x), hp);
            if (shift >= pd) shift = dadd(shift, -pd);
            r = fp::reduce(shift, m.qd, m.inv_q);
        } else {
            uint64_t shift = x + (p >> 1);
            if (shift >= p) shift -= p;
            r = fp::from_word(shift - umulhi(shift, one_s) * m.q);  // in [0, 2q)
        }
        v[k] = dadd(r, -h);
    }
}

}  // namespace ksf
}  // namespace wg
