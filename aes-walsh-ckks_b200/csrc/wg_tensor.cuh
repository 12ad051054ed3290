// One coefficient of the ciphertext tensor (ckks_mul_inplace, arith/ckks_mul.cpp:90-157), shared by the
// batched kernel (wg_batch_kernels.cuh) and the CPU emulation test.
#pragma once
#include <cstdint>

#include "wg_arith.cuh"
#include "wg_fp.cuh"

namespace wg {

// (c2, b1, a1) in place of (xa, xb): Barrett products of words as they come.
WG_HD void tensor_words(uint64_t& xa, uint64_t& xb, uint64_t ya, uint64_t yb, uint64_t& c2, const Modulus& m) {
    c2 = barrett_mul(xa, ya, m);
    const uint64_t tmp = barrett_mul(xb, ya, m);
    xb = barrett_mul(xb, yb, m);
    xa = add_mod(barrett_mul(xa, yb, m), tmp, m.q);
}

// Words that tensor_fp takes have at most one bit more than the modulus: every word below 2 q, none of
// 4 q or more.
WG_HD int tensor_shift(const Modulus& m) { return 65 - clz64(m.q); }

// The same in FP64 for moduli below fp::kNoReduce, where the four Barrett products (eight 64-bit high
// products, 3.2 SM clocks a lane) bound the kernel: |a (w / q)| < 16 q < 2^46 keeps every product exact.
// The Barrett product's one correction leaves q in place of 0 where its quotient estimate is two
// short, which takes z mod q < z q 2^-128 < 1 (q < 2^k with k <= 42, so z < 2^(2 k + 2)): for a zero
// residue alone.  Returns false for the caller to form the products in words there, and for larger
// words, whose Barrett products are congruent whatever their size.
WG_HD bool tensor_fp(uint64_t& xa, uint64_t& xb, uint64_t ya, uint64_t yb, uint64_t& c2, const Modulus& m, int shift) {
    if ((xa | xb | ya | yb) >> shift) return false;
    const double a = fp::from_word(xa), b = fp::from_word(xb);
    const fp::Factor fa = fp::key_factor(ya, m.inv_q), fb = fp::key_factor(yb, m.inv_q);
    const double aa = fp::mulmod(a, fa.w, fa.wq, m.qd), ba = fp::mulmod(b, fa.w, fa.wq, m.qd);
    const double bb = fp::mulmod(b, fb.w, fb.wq, m.qd), ab = fp::mulmod(a, fb.w, fb.wq, m.qd);
    if (aa == 0.0 || ba == 0.0 || bb == 0.0 || ab == 0.0) return false;
    c2 = fp::to_word(fp::lift(aa, m.qd));
    xb = fp::to_word(fp::lift(bb, m.qd));
    xa = fp::canonical(dadd(ab, ba), m.qd, m.inv_q);
    return true;
}

}  // namespace wg
