// Exact modular arithmetic in FP64 for moduli below 2^50.
//
// B200 issues 64 FP64 fused multiply-adds per SM and clock, and a 64-bit integer product costs
// several 32-bit multiplies plus carries: a Shoup butterfly takes about 30 integer instructions,
// the FP64 one 8.  Residues are signed integers held in doubles, any representative with
// |x| <= 2^53, so sums and differences are exact and need no correction; a product is reduced
// with the error-free pair of a product and its fused rounding error:
//
//   mulmod(a, w): h = rn(a w), l = a w - h (exact, one FMA), k = rint(a (w / q)),
//                 result (h - k q) + l = a w - k q, an integer.
//
// With |w| <= q / 2 (factors are stored centred), wq = rn(w / q) is off by at most 2^-55, so for
// |a| <= 2^52: |a wq| <= 2^51, where adding 1.5 2^52 rounds to the nearest integer (one rounding:
// it is the FMA's), and |a w - k q| <= q (1/2 + |a| 2^-55) <= 5/8 q.  h is an integer (|h| >= 2^53
// makes it one, below that it is the product), |l| <= ulp(h) / 2 <= 2^48, so |h - k q| < 2^51 and
// both remaining steps are exact.  Any |a| beyond 2^52 by a factor below 2 still gives an exact
// representative (k rounds to an even integer), only a larger one.
//
// Everything is spelled with the explicitly rounded operations of wg_arith.cuh, so neither the
// device nor the host compiler contracts or reorders a step.
#pragma once
#include <cstdint>
#include <cstring>

#include "wg_arith.cuh"

namespace wg {
namespace fp {

// Moduli that take this path.  Below kNoReduce a phase of at most 8 stages needs no reduction
// inside: its sums stay below 2^52 (see ntt::FpArith).
constexpr uint64_t kLimit = uint64_t{1} << 50;
constexpr uint64_t kNoReduce = uint64_t{1} << 42;

constexpr double kRound = 6755399441055744.0;  // 1.5 2^52: adding and subtracting it rounds to an integer
constexpr double kTwo52 = 4503599627370496.0;  // 2^52

WG_HD double bits_double(uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double d;
    std::memcpy(&d, &b, 8);
    return d;
#endif
}
WG_HD uint64_t double_bits(double d) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t b;
    std::memcpy(&b, &d, 8);
    return b;
#endif
}

// An integer below 2^52 to and from its double, without the slow conversion instructions: the
// mantissa of x + 2^52 is x.
WG_HD double from_word(uint64_t x) { return dadd(bits_double(x | 0x4330000000000000ull), -kTwo52); }
WG_HD uint64_t to_word(double x) { return double_bits(dadd(x, kTwo52)) & 0x000fffffffffffffull; }

// a w - k q for a factor (w, wq = w / q); see above.
WG_HD double mulmod(double a, double w, double wq, double q) {
    const double k = dadd(dfma(a, wq, kRound), -kRound);
    const double h = dmul(a, w);
    const double l = dfma(a, w, -h);
    return dadd(dfma(-k, q, h), l);
}

// The representative of an integer x nearest zero, |x| <= 2^53 and q >= 4: |x inv_q| <= 2^51 rounds to an
// integer as above, inv_q is off by at most 2^-53 of itself and so the quotient by at most 2^-53 |x / q| <= 1 / q
// before its rounding: |result| <= q / 2 + 1, and the subtraction is exact.
WG_HD double reduce(double x, double q, double inv_q) {
    const double k = dadd(dfma(x, inv_q, kRound), -kRound);
    return dfma(-k, q, x);
}

// The word in [0, q) of a value in (-q, q), and of any value.
WG_HD double lift(double x, double q) { return x < 0.0 ? dadd(x, q) : x; }
WG_HD uint64_t canonical(double x, double q, double inv_q) { return to_word(lift(reduce(x, q, inv_q), q)); }

// The factor pair of a residue w in [0, q), q < kLimit.
WG_HD void factor(uint64_t w, uint64_t q, double& fw, double& fwq) {
    fw = w > q / 2 ? -(double)(q - w) : (double)w;
    fwq = fw / (double)q;
}
// The factor pair of a term of a base change from a source modulus p: for a word source the factors of
// its low and high parts at bit kWordSplit.
constexpr int kWordSplit = 31;
inline void term_factor(uint64_t w, uint64_t p, uint64_t q, double& f0, double& f1) {
    factor(w, q, f0, f1);
    double unused;
    if (p >= kLimit) factor((uint64_t)(((unsigned __int128)w << kWordSplit) % q), q, f1, unused);
}
// The same on the device from the constants at hand; wq is then off by at most 2^-53, for
// |a| <= 2^51 (|result| <= 3/4 q).
WG_HD void factor_of(uint64_t w, double q, double inv_q, double& fw, double& fwq) {
    fw = from_word(w);
    if (fw > dmul(q, 0.5)) fw = dadd(fw, -q);
    fwq = dmul(fw, inv_q);
}

// Sums of Montgomery products (key inner products): each term x k, k a stored word in [0, q) (the
// factor times 2^64) and x a word below 2 q (or any |x| < 2^48 where q < kNoReduce), is formed
// without the 2^-64, which one product per sum puts back.  wq = k inv_q is off by at most 2^-52, so a term is at most 1.1 q in magnitude; sums
// of the moduli from kNoReduce up are brought to q / 2 after every fourth term.
struct Factor {
    double w, wq;
};
WG_HD Factor key_factor(uint64_t k, double inv_q) {
    const double w = from_word(k);
    return {w, dmul(w, inv_q)};
}
WG_HD double mont_sum_bound(double acc, int term, const Modulus& m) {
    return m.q >= kNoReduce && (term & 3) == 3 ? reduce(acc, m.qd, m.inv_q) : acc;
}
WG_HD double mont_sum_value(double acc, const Modulus& m) {
    if (m.q >= kNoReduce) acc = reduce(acc, m.qd, m.inv_q);
    return mulmod(acc, m.r_inv_w, m.r_inv_wq, m.qd);
}
WG_HD uint64_t mont_sum_word(double acc, const Modulus& m) { return to_word(lift(mont_sum_value(acc, m), m.qd)); }

// Sums of many products a w for moduli below kNoReduce, 4 FP64 instructions a term and one reduction
// a sum: h collects the products rounded to multiples of 2^40 (it stays in the binade of kDot, whose
// spacing that is), l the exact remainders (and any small value carried along).  Factors below 2^43
// and 2^42 give products below 2^85, so kDotTerms = 32 terms keep |h - kDot| below 2^91 and their
// remainders below 2^45.
constexpr double kDot = 1.5 * 4951760157141521099596496896.0;  // 1.5 2^92
constexpr int kDotTerms = 32;
struct Dot {
    double h, l;
    WG_HD void clear() {
        h = kDot;
        l = 0.0;
    }
    WG_HD void add(double a, double w) {
        const double t = dfma(a, w, h);
        l = dadd(l, dfma(a, w, -dadd(t, -h)));
        h = t;
    }
    // the sum so far as one term, so that kDotTerms more may follow
    WG_HD void carry(double q, double inv_q) {
        l = value(q, inv_q);
        h = kDot;
    }
    // a representative in [-q / 2, q / 2]: the quotient is at most 32 factors of 43 bits, below 2^48
    // and off by less than one part in 2^51 of itself, so the remainder of h is an integer below q
    WG_HD double value(double q, double inv_q) const {
        const double x = dadd(h, -kDot);
        const double k = dadd(dfma(x, inv_q, kRound), -kRound);
        return reduce(dadd(dfma(-k, q, x), l), q, inv_q);
    }
};

}  // namespace fp
}  // namespace wg
