// Negacyclic NTT / inverse NTT over batches of RNS limbs.
//
// Same transform as the reference's ntt_forward_dit2 / ntt_inverse_dif2 (src/math/ntt/ntt.cpp:
// 235-386): forward Cooley-Tukey with psi-folded bit-reversed twiddles (natural order in,
// bit-reversed out), inverse Gentleman-Sande with the mirrored table followed by N^-1.
// Outputs are canonical ([0, q)).
//
// Device organisation (N = 2^n, n = n1 + n2, n1 = floor(n/2)):
//   * the transform runs as two phases; the "column" phase owns the n1 high index bits, the
//     "row" phase the n2 low bits.  Forward = columns then rows, inverse = rows then columns.
//   * a CTA owns a 2048-element tile (or the whole limb for N < 2048); each thread carries 8 or 16
//     elements (the geometry's EB) through up to three or four radix-2 stages in registers per
//     round, from device memory into the first round and from the last one back;
//   * between rounds the CTA exchanges them in shared memory with one pad word every 16 words, so
//     strided 64-bit accesses stay at two wavefronts per warp;
//   * twiddles come as pairs (w, Shoup w), or (w, w / q) for the FP64 moduli below, one 16-byte load
//     each, either staged in shared memory per CTA or read from the L2-resident table directly
//     (the geometry's STAGED);
//   * grid.y indexes limbs and grid.z polynomials, so one launch covers a whole ciphertext
//     batch; each limb picks its modulus through a LimbMap (Q limbs, P limbs or a mix).
// Moduli below 2^50 (fp::kLimit) run in FP64: signed integers in doubles, exact products through
// the fused multiply-add's rounding error (wg_fp.cuh, ntt::FpArith), 8 FP64 instructions a
// butterfly against about 30 integer ones; between the phases a limb holds the doubles' bits.
// Larger moduli use Harvey/Shoup butterflies on words with lazy ranges: forward values stay in
// [0, 4q) (or, for moduli below 2^58, grow by at most 2q per stage without reduction, see
// kLazyForwardLimit), inverse in [0, 2q).  The last phase canonicalises (forward) or scales by
// N^-1 (inverse), so both give the same words.
// Every geometry performs the same butterflies on the same values, so all of them give the
// same words; which one runs is chosen per (direction, phase) by timing them on the device
// when a context is created (ntt_autotune).
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "wg_internal.hpp"
#include "wg_ntt.cuh"

namespace wg {
namespace {
using namespace ntt;

// The rounds of one phase on a thread's elements, exchanged through `sm` in between: v enters in the
// first round's places and leaves in the last one's.  `sm` may still be read by others on entry.
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL, int RD, class Arith>
__device__ __forceinline__ void ntt_round(uint64_t* sm, typename Arith::V* v, int sub, int o, int tile,
                                          const Arith& ar, const TwPair* tw) {
    if constexpr (RD > 0) {
        __syncthreads();
        Round<LOGN, FWD, COLS, EB, STAGED, RD - 1, TL>::template scatter<Arith>(sm, sub, o, v);
        __syncthreads();
        Round<LOGN, FWD, COLS, EB, STAGED, RD, TL>::template gather<Arith>(sm, sub, o, v);
    }
    Round<LOGN, FWD, COLS, EB, STAGED, RD, TL>::stages(v, sub, o, tile, ar, tw);
}
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL, class Arith, int... RD>
__device__ __forceinline__ void ntt_rounds(std::integer_sequence<int, RD...>, uint64_t* sm, typename Arith::V* v,
                                           int sub, int o, int tile, const Arith& ar, const TwPair* tw) {
    (ntt_round<LOGN, FWD, COLS, EB, STAGED, TL, RD>(sm, v, sub, o, tile, ar, tw), ...);
}

// A thread's elements of a round to and from one limb.  A run of consecutive words (the row phase's
// last bits) goes in whole 32-byte sectors where the limb is aligned to them: a word at a time, every
// access of a warp would touch 32 sectors for a quarter of each.
template <class R>
__device__ __forceinline__ void load_words(const uint64_t* __restrict__ p, uint64_t* w) {
    if (R::RUN && (reinterpret_cast<uintptr_t>(p) & 31) == 0) {
#pragma unroll
        for (int j = 0; j < R::E; j += 4)
            asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];\n"
                         : "=l"(w[j]), "=l"(w[j + 1]), "=l"(w[j + 2]), "=l"(w[j + 3])
                         : "l"(p + j)
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < R::E; ++j) w[j] = p[R::limb_step(j)];
    }
}
template <class R>
__device__ __forceinline__ void store_words(uint64_t* __restrict__ p, const uint64_t* w) {
    if (R::RUN && (reinterpret_cast<uintptr_t>(p) & 31) == 0) {
#pragma unroll
        for (int j = 0; j < R::E; j += 4)
            asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};\n" ::"l"(p + j), "l"(w[j]), "l"(w[j + 1]),
                         "l"(w[j + 2]), "l"(w[j + 3])
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < R::E; ++j) p[R::limb_step(j)] = w[j];
    }
}

template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED>
constexpr size_t smem_bytes() {
    using P = Phase<LOGN, FWD, COLS, EB, STAGED>;
    return 8 * (size_t)(P::TILE + P::TILE / 16) + (STAGED ? 16 * (size_t)P::TW : 0);
}

// CTAs per SM: 8-residue rounds fit 64 registers (256 threads), 16-residue ones get up to 128 (128 threads).
constexpr int kMinBlocks = 4;

// The twiddle pairs a CTA reads, copied to shared memory in twiddle_src order.
template <int LOGN, bool FWD, bool COLS, int EB>
__device__ __forceinline__ void stage_twiddles(const TwPair* __restrict__ tw, TwPair* tw_s, int tile, int t) {
    using P = Phase<LOGN, FWD, COLS, EB, true>;
    const ulonglong2* src2 = reinterpret_cast<const ulonglong2*>(tw);
    ulonglong2* dst2 = reinterpret_cast<ulonglong2*>(tw_s);
    if (COLS) {
        for (int e = t; e < P::TW; e += P::THREADS) dst2[e] = __ldg(src2 + e);
    } else {
        // row-stage k: SUBS * 2^k contiguous table entries
#pragma unroll
        for (int k = 0; k < P::MB; ++k) {
            const int cnt = P::SUBS << k;
            const int dst = P::SUBS * ((1 << k) - 1);
            const size_t src = ((size_t)1 << (P::NB1 + k)) + (size_t)tile * cnt;
            for (int e = t; e < cnt; e += P::THREADS) dst2[dst + e] = __ldg(src2 + src + e);
        }
    }
}

// Addressing of one limb: either a strided batch (blockIdx.y = limb, blockIdx.z = polynomial,
// modulus from a LimbMap) or an entry of a job table (blockIdx.y + 65535 * blockIdx.z).  The
// first phase may read from a different buffer than it writes (src -> dst); the second phase
// works in place on dst.
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, bool TABLE>
__global__ void __launch_bounds__(Phase<LOGN, FWD, COLS, EB, STAGED>::THREADS, kMinBlocks)
    k_ntt_phase(uint64_t* __restrict__ data, size_t poly_stride, LimbMap map, const NttJob* __restrict__ jobs,
                int njobs, const Modulus* __restrict__ mods, const TwPair* __restrict__ tw_base,
                const TwPair* __restrict__ tw_words) {
    using P = Phase<LOGN, FWD, COLS, EB, STAGED>;
    constexpr int N = P::N;
    constexpr int E = P::E;
    constexpr bool FIRST = FWD ? COLS : !COLS;
    extern __shared__ __align__(16) uint64_t smem[];
    uint64_t* sm = smem;                                                       // exchange tile, padded
    TwPair* tw_s = reinterpret_cast<TwPair*>(smem + P::TILE + P::TILE / 16);  // staged twiddles

    const uint64_t* xin;
    uint64_t* x;
    int mi;
    bool words = false;
    if (TABLE) {
        const int j = blockIdx.y + 65535 * blockIdx.z;
        if (j >= njobs) return;
        const NttJob job = jobs[j];
        x = job.dst;
        xin = FIRST ? job.src : job.dst;
        mi = job.mod;
        words = !FWD && !COLS && job.words != 0;
    } else {
        const int limb = blockIdx.y;
        x = data + (size_t)blockIdx.z * poly_stride + (size_t)limb * N;
        xin = x;
        mi = map(limb);
    }
    const Modulus m = mods[mi];
    const bool fp64 = m.q < fp::kLimit && !words;
    const TwPair* tw = words ? tw_words + (size_t)mi * N : tw_base + (size_t)mi * 2 * N + (FWD ? 0 : N);
    const int tile = blockIdx.x;
    const int t = threadIdx.x, sub = P::sub_of(t), o = P::o_of(t);
    using Begin = Round<LOGN, FWD, COLS, EB, STAGED, 0>;
    using End = Round<LOGN, FWD, COLS, EB, STAGED, P::ROUNDS - 1>;
    uint64_t w[E];
    load_words<Begin>(xin + tile_offset<LOGN, FWD, COLS, EB, STAGED>(tile, Begin::element(sub, o)), w);
    if (STAGED) {
        stage_twiddles<LOGN, FWD, COLS, EB>(tw, tw_s, tile, t);
        __syncthreads();
    }
    const TwPair* twr = STAGED ? tw_s : tw;
    constexpr auto rounds = std::make_integer_sequence<int, P::ROUNDS>{};
    if (fp64) {
        double v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = fp::bits_double(fp_load(FIRST, w[j], m));
        ntt_rounds<LOGN, FWD, COLS, EB, STAGED, kMaxTile>(rounds, sm, v, sub, o, tile, fp_arith(m), twr);
#pragma unroll
        for (int j = 0; j < E; ++j) w[j] = fp_store(P::LAST, FWD, fp::double_bits(v[j]), m);
    } else {
        // forward transforms under kLazyForwardLimit skip the per-butterfly reduction
        if (FWD && m.q < kLazyForwardLimit)
            ntt_rounds<LOGN, FWD, COLS, EB, STAGED, kMaxTile>(rounds, sm, w, sub, o, tile, WordArith<FWD>{m.q}, twr);
        else
            ntt_rounds<LOGN, FWD, COLS, EB, STAGED, kMaxTile>(rounds, sm, w, sub, o, tile, WordArith<false>{m.q}, twr);
#pragma unroll
        for (int j = 0; j < E; ++j) w[j] = word_store(P::LAST, FWD, w[j], m);
    }
    store_words<End>(x + tile_offset<LOGN, FWD, COLS, EB, STAGED>(tile, End::element(sub, o)), w);
}

// A whole transform of one limb per cluster (Whole, wg_ntt.cuh): both phases' rounds with the results
// of the first handed over in distributed shared memory, so a limb crosses device memory once each
// way instead of twice and a small batch pays one launch.
// `between` is applied to the first phase's values on their way to the second's tiles.
template <int LOGN, bool FWD, class Arith, class Between>
__device__ __forceinline__ void whole_transform(uint64_t* first, uint64_t* second, typename Arith::V* v, int tile, int t,
                                                const Arith& ar, const TwPair* tw, Between between) {
    using W = Whole<LOGN>;
    using P1 = typename W::template Ph<FWD, FWD>;
    using P2 = typename W::template Ph<FWD, !FWD>;
    using End = Round<LOGN, FWD, FWD, 3, false, P1::ROUNDS - 1, W::TL>;
    using Begin = Round<LOGN, FWD, !FWD, 3, false, 0, W::TL>;
    ntt_rounds<LOGN, FWD, FWD, 3, false, W::TL>(std::make_integer_sequence<int, P1::ROUNDS>{}, first, v, P1::sub_of(t),
                                                P1::o_of(t), tile, ar, tw);
    if (W::CTAS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");  // every CTA has started
    const int e0 = End::element(P1::sub_of(t), P1::o_of(t));
#pragma unroll
    for (int j = 0; j < End::E; ++j) {
        const HandOver h = hand_over<LOGN, FWD>(tile, e0 + End::tile_step(j));
        const uint64_t w = between(Arith::bits(v[j]));
        if (W::CTAS > 1) {
            const unsigned local = (unsigned)__cvta_generic_to_shared(second + pad16(h.at));
            unsigned remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local), "r"(h.cta));
            asm volatile("st.shared::cluster.u64 [%0], %1;\n" ::"r"(remote), "l"(w) : "memory");
        } else {
            second[pad16(h.at)] = w;
        }
    }
    if (W::CTAS > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    } else {
        __syncthreads();
    }
    Begin::template gather<Arith>(second, P2::sub_of(t), P2::o_of(t), v);
    // no CTA writes to `second` any more, but its own threads still read: the rounds exchange in `first`
    ntt_rounds<LOGN, FWD, !FWD, 3, false, W::TL>(std::make_integer_sequence<int, P2::ROUNDS>{}, first, v, P2::sub_of(t),
                                                 P2::o_of(t), tile, ar, tw);
}

template <int LOGN>
constexpr size_t whole_smem() {
    return 2 * 8 * (size_t)Whole<LOGN>::PAD;
}

template <int LOGN, bool FWD, bool TABLE>
__global__ void __launch_bounds__(Whole<LOGN>::template Ph<FWD, true>::THREADS,
                                  1024 / Whole<LOGN>::template Ph<FWD, true>::THREADS)
    k_ntt_whole(uint64_t* __restrict__ data, size_t poly_stride, LimbMap map, const NttJob* __restrict__ jobs, int njobs,
                const Modulus* __restrict__ mods, const TwPair* __restrict__ tw_base) {
    using W = Whole<LOGN>;
    using P1 = typename W::template Ph<FWD, FWD>;
    using P2 = typename W::template Ph<FWD, !FWD>;
    using Begin = Round<LOGN, FWD, FWD, 3, false, 0, W::TL>;
    using End = Round<LOGN, FWD, !FWD, 3, false, P2::ROUNDS - 1, W::TL>;
    constexpr int E = 8;
    extern __shared__ __align__(16) uint64_t smem[];
    uint64_t* first = smem;
    uint64_t* second = smem + W::PAD;
    const uint64_t* xin;
    uint64_t* x;
    int mi;
    if (TABLE) {
        const int j = blockIdx.y + 65535 * blockIdx.z;
        if (j >= njobs) return;  // the same for every CTA of a cluster
        const NttJob job = jobs[j];
        x = job.dst;
        xin = job.src;
        mi = job.mod;
    } else {
        const int limb = blockIdx.y;
        x = data + (size_t)blockIdx.z * poly_stride + (size_t)limb * W::N;
        xin = x;
        mi = map(limb);
    }
    if (W::CTAS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
    const Modulus m = mods[mi];
    const TwPair* tw = tw_base + (size_t)mi * 2 * W::N + (FWD ? 0 : W::N);
    const int tile = blockIdx.x, t = threadIdx.x;
    uint64_t w[E];
    load_words<Begin>(
        xin + tile_offset<LOGN, FWD, FWD, 3, false, W::TL>(tile, Begin::element(P1::sub_of(t), P1::o_of(t))), w);
    if (m.q < fp::kLimit) {
        double v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = fp::bits_double(fp_load(true, w[j], m));
        whole_transform<LOGN, FWD>(first, second, v, tile, t, fp_arith(m), tw,
                                   [&](uint64_t b) { return fp_store(false, FWD, b, m); });
#pragma unroll
        for (int j = 0; j < E; ++j) w[j] = fp_store(true, FWD, fp::double_bits(v[j]), m);
    } else {
        const auto same = [](uint64_t b) { return b; };
        if (FWD && m.q < kLazyForwardLimit)
            whole_transform<LOGN, FWD>(first, second, w, tile, t, WordArith<FWD>{m.q}, tw, same);
        else
            whole_transform<LOGN, FWD>(first, second, w, tile, t, WordArith<false>{m.q}, tw, same);
#pragma unroll
        for (int j = 0; j < E; ++j) w[j] = word_store(true, FWD, w[j], m);
    }
    store_words<End>(
        x + tile_offset<LOGN, FWD, !FWD, 3, false, W::TL>(tile, End::element(P2::sub_of(t), P2::o_of(t))), w);
}

template <int LOGN, bool FWD, bool TABLE>
void launch_whole(const Context& c, uint64_t* data, int limbs, int polys, size_t stride, LimbMap map,
                  const NttJob* jobs, int njobs, cudaStream_t s) {
    using W = Whole<LOGN>;
    static_assert(whole_smem<LOGN>() <= size_t{48} << 10, "no opt-in");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = TABLE ? dim3(W::CTAS, njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535)
                        : dim3(W::CTAS, limbs, polys);
    cfg.blockDim = dim3(W::template Ph<FWD, true>::THREADS);
    cfg.dynamicSmemBytes = whole_smem<LOGN>();
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = W::CTAS;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    // algorithmic bytes: every residue read once and written once
    Probe probe(kClsNtt, 16.0 * W::N * (TABLE ? njobs : (double)limbs * polys), s);
    check_cuda(cudaLaunchKernelEx(&cfg, k_ntt_whole<LOGN, FWD, TABLE>, data, stride, map, jobs, njobs,
                                  (const Modulus*)c.d_mod, c.twiddles(3)),
               "ntt launch");
}

template <int LOGN>
void whole_dispatch(const Context& c, uint64_t* data, int limbs, int polys, size_t stride, LimbMap map,
                    const NttJob* jobs, int njobs, bool fwd, cudaStream_t s) {
    if (jobs) {
        if (fwd) launch_whole<LOGN, true, true>(c, data, limbs, polys, stride, map, jobs, njobs, s);
        else launch_whole<LOGN, false, true>(c, data, limbs, polys, stride, map, jobs, njobs, s);
    } else {
        if (fwd) launch_whole<LOGN, true, false>(c, data, limbs, polys, stride, map, jobs, njobs, s);
        else launch_whole<LOGN, false, false>(c, data, limbs, polys, stride, map, jobs, njobs, s);
    }
}

// The forward row phase of one job-table limb with an element-wise epilogue (NttEpiJob): the
// same rounds and final reduction as k_ntt_phase<LOGN, true, false, ...>, then the epilogue in
// place of the store.  The epilogue's operands (acc, in: the tile's contiguous words) are
// copied into shared memory with cp.async when the block starts, so their loads overlap the
// rounds instead of stalling the final step; out may alias acc or in, since each word is read
// and written by this block only.
template <int LOGN, int EB, bool STAGED>
constexpr size_t rows_epi_smem() {
    using P = Phase<LOGN, true, false, EB, STAGED>;
    return smem_bytes<LOGN, true, false, EB, STAGED>() + 2 * 8 * (size_t)P::TILE;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(gmem) : "memory");
}

template <int LOGN, int EB, bool STAGED>
__global__ void __launch_bounds__(Phase<LOGN, true, false, EB, STAGED>::THREADS, kMinBlocks)
    k_ntt_rows_epi(const NttEpiJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods,
                   const TwPair* __restrict__ tw_base) {
    using P = Phase<LOGN, true, false, EB, STAGED>;
    constexpr int N = P::N;
    constexpr int E = P::E;
    extern __shared__ __align__(16) uint64_t smem[];
    uint64_t* sm = smem;
    TwPair* tw_s = reinterpret_cast<TwPair*>(smem + P::TILE + P::TILE / 16);
    uint64_t* acc_s = smem + smem_bytes<LOGN, true, false, EB, STAGED>() / 8;
    uint64_t* in_s = acc_s + P::TILE;
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    const NttEpiJob job = jobs[j];
    const int mi = job.mod;
    const Modulus m = mods[mi];
    const TwPair* tw = tw_base + (size_t)mi * 2 * N;
    const int tile = blockIdx.x;
    const int t = threadIdx.x;
    // the row tile is P::TILE contiguous words at tile * TILE: 16-byte copies when the operand
    // limbs are 16-byte aligned (they start on a word; tile * TILE keeps any 16-byte alignment),
    // 8-byte copies otherwise
    const size_t base = (size_t)tile * P::TILE;
    const bool need_acc = job.kind == kEpiCombine;
    const bool need_in = job.kind == kEpiRescale || job.c0 != 0;
    const uintptr_t align = (need_acc ? reinterpret_cast<uintptr_t>(job.acc) : 0) |
                            (need_in ? reinterpret_cast<uintptr_t>(job.in) : 0);
    if ((align & 15) == 0) {
        for (int c = t; c < P::TILE / 2; c += P::THREADS) {
            if (need_acc) cp_async16(acc_s + 2 * c, job.acc + base + 2 * c);
            if (need_in) cp_async16(in_s + 2 * c, job.in + base + 2 * c);
        }
    } else {
        for (int e = t; e < P::TILE; e += P::THREADS) {
            if (need_acc) cp_async8(acc_s + e, job.acc + base + e);
            if (need_in) cp_async8(in_s + e, job.in + base + e);
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    using Begin = Round<LOGN, true, false, EB, STAGED, 0>;
    using End = Round<LOGN, true, false, EB, STAGED, P::ROUNDS - 1>;
    const int sub = P::sub_of(t), o = P::o_of(t);
    uint64_t w[E];
    load_words<Begin>(job.data + base + Begin::element(sub, o), w);
    if (STAGED) {
        stage_twiddles<LOGN, true, false, EB>(tw, tw_s, tile, t);
        __syncthreads();
    }
    const TwPair* twr = STAGED ? tw_s : tw;
    constexpr auto rounds = std::make_integer_sequence<int, P::ROUNDS>{};
    const bool fp64 = m.q < fp::kLimit;
    // the last round's values through the tile once more, so that the epilogue's accesses are
    // consecutive over a warp as its operands' copies are
    if (fp64) {
        double v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = fp::bits_double(w[j]);
        ntt_rounds<LOGN, true, false, EB, STAGED, kMaxTile>(rounds, sm, v, sub, o, tile, fp_arith(m), twr);
        __syncthreads();
        End::template scatter<FpArith>(sm, sub, o, v);
    } else {
        if (m.q < kLazyForwardLimit)
            ntt_rounds<LOGN, true, false, EB, STAGED, kMaxTile>(rounds, sm, w, sub, o, tile, WordArith<true>{m.q}, twr);
        else
            ntt_rounds<LOGN, true, false, EB, STAGED, kMaxTile>(rounds, sm, w, sub, o, tile, WordArith<false>{m.q}, twr);
        __syncthreads();
        End::template scatter<WordArith<false>>(sm, sub, o, w);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    const FpEpilogue c = fp64 ? fp_epilogue(job, m) : FpEpilogue{};
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const int e = t + k * P::THREADS;
        const uint64_t x = sm[pad16(e)], acc = need_acc ? acc_s[e] : 0, in = need_in ? in_s[e] : 0;
        job.out[base + e] = fp64 ? fp_epilogue_value(job, c, acc, in, x, m)
                                 : epilogue_value(job, acc, in, word_store(true, true, x, m), m.q);
    }
}

// The forward row phase of a switch's digits with the key inner product on it, for one QP limb's
// row tile: a digit's transformed words meet the key words in the registers of the last round, where a
// thread has 8 consecutive coefficients, and only the two accumulators are stored; an
// accumulator's P limb goes straight on through its inverse row phase, whose first round has the
// thread's same 8 coefficients.  Against the separate launches a digit limb is read once instead of
// written and read again twice over, and a switch takes two launches less.  The switches of a job
// follow one another, so a tile's key words (parts x 32 KiB) come from L1 after the first.
// One rotation takes 95 us, 104 with the separate launches; 64 mixed operations 4.23 ms against 4.49; the
// 16 S-boxes of an XBOOT SubBytes layer 84.9 ms against 89.6.  Two blocks of 256 threads an SM (128
// registers: the sums, the residues and the next digit's): latency, not the FP64 pipe, bounds it.  Limbs of
// word moduli spill some of them here and still gain: with theirs in the separate launches the
// transforms and key products of a Walsh AES take 334 ms, with them 325, of 64 mixed operations 2.08 and
// 1.89.
template <int LOGN>
struct RowsMac {
    using P = Phase<LOGN, true, false, 3, false>;
    using Begin = Round<LOGN, true, false, 3, false, 0>;
    using End = Round<LOGN, true, false, 3, false, P::ROUNDS - 1>;
    using InvEnd = Round<LOGN, false, false, 3, false, P::ROUNDS - 1>;
    static constexpr auto rounds() { return std::make_integer_sequence<int, P::ROUNDS>{}; }
    static constexpr size_t smem() { return 8 * (size_t)(P::TILE + P::TILE / 16); }
};
// One switch (c) of a job: Sums is the modulus's arithmetic (MacSumsFp, MacSumsWords), `fwd` and `inv` the
// rounds' (FP64: one for both).  AHEAD: the next digit is loaded before the products with this one's key words.
template <int LOGN, bool AHEAD, class Sums, class Fwd, class Inv>
__device__ __forceinline__ void rows_mac(uint64_t* sm, const MacGroupJob* j, int c, const Modulus& m, bool rows,
                                         size_t at, size_t key_at, size_t key_stride, int own_part, size_t T, int tile,
                                         int sub, int o, const TwPair* tw, const Fwd& fwd, const Inv& inv) {
    using R = RowsMac<LOGN>;
    const size_t N = R::P::N;
    const int eb = R::Begin::element(sub, o), ee = R::End::element(sub, o), parts = j->parts;
    const uint64_t* digits = j->digits[c] + at + eb;
    const uint64_t* own = j->key_term[c] + at + ee;
    uint64_t w[8], k8[8];
    // (the word sums leave no registers for the two pointers: read again from the job)
    auto fetch = [&](int p) {
        if (p == own_part)
            load_words<typename R::End>(AHEAD ? own : j->key_term[c] + at + ee, w);
        else
            load_words<typename R::Begin>((AHEAD ? digits : j->digits[c] + at + eb) + p * j->part_stride, w);
    };
    Sums sums;
    sums.clear();
    typename Sums::V ahead[8], *v;  // the residues: beside the next digit's words, or in their place
    if constexpr (AHEAD)
        v = ahead;
    else
        v = w;
    if (AHEAD) fetch(0);
    for (int p = 0; p < parts; ++p) {
        if (!AHEAD) fetch(p);
        if (p == own_part) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = Sums::own(w[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = Sums::digit(w[k]);
            ntt_rounds<LOGN, true, false, 3, false, kMaxTile>(R::rounds(), sm, v, sub, o, tile, fwd, tw);
            Sums::transformed(v, m);
        }
        if (AHEAD && p + 1 < parts) fetch(p + 1);
        const uint64_t* key = j->key + p * 2 * key_stride + key_at + ee;
        load_words<typename R::End>(key, k8);
        sums.add(0, v, k8, p, m);
        load_words<typename R::End>(key + key_stride, k8);
        sums.add(1, v, k8, p, m);
    }
#pragma unroll
    for (int poly = 0; poly < 2; ++poly) {
        uint64_t* out = j->acc[c] + poly * T * N + at;
        if (!AHEAD || rows) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = sums.value(poly, k, m);
        }
        if (rows) {
            ntt_rounds<LOGN, false, false, 3, false, kMaxTile>(R::rounds(), sm, v, sub, o, tile, inv, tw + N);
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = Sums::row_word(v[k], m);
            store_words<typename R::InvEnd>(out + R::InvEnd::element(sub, o), w);
        } else {
            if constexpr (AHEAD) {
#pragma unroll
                for (int k = 0; k < 8; ++k) w[k] = sums.word(poly, k, m);
            }
            store_words<typename R::End>(out + ee, w);  // (word sums: v is w, and the value the word)
        }
    }
}

template <int LOGN, bool WORDS>
__global__ void __launch_bounds__(RowsMac<LOGN>::P::THREADS, 2)
    k_rows_mac(const MacGroupJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods, int nq,
               const TwPair* __restrict__ tw_base) {
    using P = typename RowsMac<LOGN>::P;
    const int jn = blockIdx.y + 65535 * blockIdx.z;
    if (jn >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const MacGroupJob* j = jobs + jn;
    const int i = j->i, L = j->L, K = j->K, tile = blockIdx.x, t = threadIdx.x;
    const bool is_p = i >= L;
    const int mi = is_p ? nq + (i - L) : i;
    const Modulus m = mods[mi];
    const TwPair* tw = tw_base + (size_t)mi * 2 * P::N;
    const size_t key_limbs = (size_t)j->key_level + 1 + K, key_stride = key_limbs * P::N;
    const size_t klimb = is_p ? (size_t)j->key_level + 1 + (i - L) : (size_t)i;
    const size_t at = (size_t)i * P::N + (size_t)tile * P::TILE, key_at = klimb * P::N + (size_t)tile * P::TILE;
    const int own_part = is_p ? -1 : i / j->alpha, sub = P::sub_of(t), o = P::o_of(t);
    const size_t T = L + K;
    for (int c = 0; c < j->n; ++c) {
        if (!WORDS || m.q < fp::kLimit) {
            const FpArith ar = fp_arith(m);
            rows_mac<LOGN, true, MacSumsFp>(smem, j, c, m, is_p, at, key_at, key_stride, own_part, T, tile, sub, o, tw, ar, ar);
        } else if (m.q < kLazyForwardLimit) {
            rows_mac<LOGN, false, MacSumsWords>(smem, j, c, m, is_p, at, key_at, key_stride, own_part, T, tile, sub, o, tw,
                                                WordArith<true>{m.q}, WordArith<false>{m.q});
        } else {
            const WordArith<false> ar{m.q};
            rows_mac<LOGN, false, MacSumsWords>(smem, j, c, m, is_p, at, key_at, key_stride, own_part, T, tile, sub, o, tw, ar,
                                                ar);
        }
    }
}

template <int LOGN>
void launch_rows_mac(const Context& c, const MacGroupJob* jobs, int njobs, cudaStream_t s) {
    using P = typename RowsMac<LOGN>::P;
    const dim3 grid(P::N / P::TILE, njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    if (c.word_moduli)
        k_rows_mac<LOGN, true><<<grid, P::THREADS, RowsMac<LOGN>::smem(), s>>>(jobs, njobs, c.d_mod, (int)c.nq,
                                                                               c.twiddles(3));
    else
        k_rows_mac<LOGN, false><<<grid, P::THREADS, RowsMac<LOGN>::smem(), s>>>(jobs, njobs, c.d_mod, (int)c.nq,
                                                                                c.twiddles(3));
}

template <int LOGN, int EB, bool STAGED>
void launch_rows_epi(const Context& c, const NttEpiJob* jobs, int njobs, cudaStream_t s) {
    using P = Phase<LOGN, true, false, EB, STAGED>;
    constexpr size_t sm = rows_epi_smem<LOGN, EB, STAGED>();
    allow_shared<k_ntt_rows_epi<LOGN, EB, STAGED>>(c.device, sm);
    const dim3 grid(P::N / P::TILE, njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_ntt_rows_epi<LOGN, EB, STAGED><<<grid, P::THREADS, sm, s>>>(jobs, njobs, c.d_mod, c.twiddles(EB));
}

template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED>
void launch_geom(const Context& c, uint64_t* data, int limbs, int polys, size_t stride, LimbMap map,
                 const NttJob* jobs, int njobs, cudaStream_t s) {
    using P = Phase<LOGN, FWD, COLS, EB, STAGED>;
    constexpr size_t sm = smem_bytes<LOGN, FWD, COLS, EB, STAGED>();
    const TwPair* tw = c.twiddles(COLS ? 3 : EB);  // column phases read the part that all orders share
    if (jobs) {
        allow_shared<k_ntt_phase<LOGN, FWD, COLS, EB, STAGED, true>>(c.device, sm);
        const dim3 grid(P::N / P::TILE, njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
        // algorithmic bytes: every residue read once and written once per transform, i.e. 8 B
        // per residue for each of the two phases (16 N B per limb-transform)
        Probe probe(kClsNtt, 8.0 * P::N * njobs, s);
        k_ntt_phase<LOGN, FWD, COLS, EB, STAGED, true><<<grid, P::THREADS, sm, s>>>(nullptr, 0, map, jobs, njobs,
                                                                                   c.d_mod, tw,
                                                                                   c.word_twiddles(COLS ? 3 : EB));
    } else {
        allow_shared<k_ntt_phase<LOGN, FWD, COLS, EB, STAGED, false>>(c.device, sm);
        const dim3 grid(P::N / P::TILE, limbs, polys);
        Probe probe(kClsNtt, 8.0 * P::N * limbs * polys, s);
        k_ntt_phase<LOGN, FWD, COLS, EB, STAGED, false><<<grid, P::THREADS, sm, s>>>(data, stride, map, nullptr, 0,
                                                                                    c.d_mod, tw, nullptr);
    }
}

// One phase with the geometry `variant` (kNttGeometries order).
template <int LOGN, bool FWD, bool COLS>
void launch_phase(const Context& c, int variant, uint64_t* data, int limbs, int polys, size_t stride, LimbMap map,
                  const NttJob* jobs, int njobs, cudaStream_t s) {
    switch (variant) {
        case 0: launch_geom<LOGN, FWD, COLS, 3, true>(c, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 1: launch_geom<LOGN, FWD, COLS, 3, false>(c, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 2: launch_geom<LOGN, FWD, COLS, 4, true>(c, data, limbs, polys, stride, map, jobs, njobs, s); break;
        default: launch_geom<LOGN, FWD, COLS, 4, false>(c, data, limbs, polys, stride, map, jobs, njobs, s); break;
    }
}

template <int LOGN>
void run_phase(const Context& c, bool fwd, bool cols, int variant, uint64_t* data, int limbs, int polys, size_t stride,
               LimbMap map, const NttJob* jobs, int njobs, cudaStream_t s) {
    if (fwd) {
        if (cols) launch_phase<LOGN, true, true>(c, variant, data, limbs, polys, stride, map, jobs, njobs, s);
        else launch_phase<LOGN, true, false>(c, variant, data, limbs, polys, stride, map, jobs, njobs, s);
    } else {
        if (cols) launch_phase<LOGN, false, true>(c, variant, data, limbs, polys, stride, map, jobs, njobs, s);
        else launch_phase<LOGN, false, false>(c, variant, data, limbs, polys, stride, map, jobs, njobs, s);
    }
}

void phase_dispatch(const Context& c, bool fwd, bool cols, int variant, uint64_t* data, int limbs, int polys,
                    size_t stride, LimbMap map, const NttJob* jobs, int njobs, cudaStream_t s) {
    switch (c.logN) {
        case 10: run_phase<10>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 11: run_phase<11>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 12: run_phase<12>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 13: run_phase<13>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 14: run_phase<14>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 15: run_phase<15>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        case 16: run_phase<16>(c, fwd, cols, variant, data, limbs, polys, stride, map, jobs, njobs, s); break;
        default: fail(kInvalid, "ntt: ring degree must be 2^10 .. 2^16");
    }
}

// The geometry of one phase over `words` residues: the caller's where it is pinned, else by the tuned one.
int phase_geometry(const Context& c, int direction, bool cols, size_t words) {
    const int v = c.ntt_variant[direction][cols ? 1 : 0];
    return c.ntt_pinned[direction] >> (cols ? 1 : 0) & 1 ? v : launch_geometry(v, cols, words, c.sm_count, c.word_moduli);
}

void dispatch(const Context& c, uint64_t* data, int limbs, int polys, size_t stride, LimbMap map,
              const NttJob* jobs, int njobs, bool fwd, cudaStream_t s) {
    if (jobs ? njobs <= 0 : (limbs <= 0 || polys <= 0)) return;
    if (!jobs && (polys > 65535 || limbs > 65535)) fail(kInvalid, "ntt: too many limbs or polynomials in one batch");
    const int d = fwd ? 0 : 1;
    const size_t transforms = jobs ? (size_t)njobs : limbs * (size_t)polys, words = transforms * c.N;
    if (!c.ntt_pinned[d] && whole_launch(c.logN, transforms, c.sm_count, c.word_moduli)) {
        switch (c.logN) {
            case 10: whole_dispatch<10>(c, data, limbs, polys, stride, map, jobs, njobs, fwd, s); break;
            case 11: whole_dispatch<11>(c, data, limbs, polys, stride, map, jobs, njobs, fwd, s); break;
            case 12: whole_dispatch<12>(c, data, limbs, polys, stride, map, jobs, njobs, fwd, s); break;
            case 13: whole_dispatch<13>(c, data, limbs, polys, stride, map, jobs, njobs, fwd, s); break;
            default: whole_dispatch<14>(c, data, limbs, polys, stride, map, jobs, njobs, fwd, s); break;
        }
        return;
    }
    // forward: columns then rows; inverse: rows then columns
    const bool first_cols = fwd;
    phase_dispatch(c, fwd, first_cols, phase_geometry(c, d, first_cols, words), data, limbs, polys, stride, map, jobs,
                   njobs, s);
    phase_dispatch(c, fwd, !first_cols, phase_geometry(c, d, !first_cols, words), data, limbs, polys, stride, map,
                   jobs, njobs, s);
    check_cuda(cudaGetLastError(), "ntt launch");
}

// Tuned choices per (device, ring degree, share of word moduli in quarters, rounded up), shared by the
// process's contexts: FP64 and integer limbs favour different geometries, and a chain's launches mix
// them as its timing batch does.
struct TuneKey {
    int device, logN, words;
    bool operator<(const TuneKey& o) const {
        return std::tie(device, logN, words) < std::tie(o.device, o.logN, o.words);
    }
};
TuneKey tune_key(const Context& c) {
    const auto n = std::count_if(c.mods.begin(), c.mods.end(), [](const Modulus& m) { return m.q >= fp::kLimit; });
    return {c.device, c.logN, (int)((4 * n + c.mods.size() - 1) / c.mods.size())};
}
std::mutex g_tune_mutex;
std::map<TuneKey, NttTuning> g_tuned;

void take_tuning(Context& c) {
    bool rows16 = false;
    for (int d = 0; d < 2; ++d)
        for (int p = 0; p < 2; ++p) {
            c.ntt_variant[d][p] = c.tuning.chosen[d][p];
            rows16 |= p == 0 && c.tuning.chosen[d][p] >= 2;
        }
    c.rows16(rows16);
}

}  // namespace

void ntt_forward(const Context& c, uint64_t* data, int limbs, int polys, size_t poly_stride, LimbMap map,
                 cudaStream_t s) {
    dispatch(c, data, limbs, polys, poly_stride, map, nullptr, 0, true, s);
}

void ntt_inverse(const Context& c, uint64_t* data, int limbs, int polys, size_t poly_stride, LimbMap map,
                 cudaStream_t s) {
    dispatch(c, data, limbs, polys, poly_stride, map, nullptr, 0, false, s);
}

void ntt_jobs(const Context& c, const NttJob* d_jobs, int njobs, bool forward, cudaStream_t s) {
    dispatch(c, nullptr, 0, 0, 0, LimbMap{0, 0, 0}, d_jobs, njobs, forward, s);
}

void ntt_jobs_phase(const Context& c, const NttJob* d_jobs, int njobs, bool forward, bool cols, cudaStream_t s) {
    if (njobs <= 0) return;
    phase_dispatch(c, forward, cols, phase_geometry(c, forward ? 0 : 1, cols, njobs * c.N), nullptr, 0, 0, 0,
                   LimbMap{0, 0, 0}, d_jobs, njobs, s);
    check_cuda(cudaGetLastError(), "ntt launch");
}

// Two switches a job share the key words in L1 where that leaves eight waves of two blocks an SM; longer
// jobs lose in the last wave what they read less (XBOOT S-box layer: 34.8, 33.5 and 32.9 ms at 1, 2 and
// 4 a job, a bootstrap's 13.2, 13.2 and 13.4; a Walsh AES's 339, 340 and 367 at 1, 2 and 8).
int rows_mac_group(const Context& c, size_t switches, size_t T) {
    const size_t tiles = std::max<size_t>(1, c.N / kMaxTile);
    return switches * T * tiles >= 16 * (size_t)c.sm_count ? 2 : 1;
}

void rows_mac_jobs(const Context& c, const MacGroupJob* d_jobs, int njobs, double bytes, cudaStream_t s) {
    if (njobs <= 0) return;
    Probe probe(kClsKeyMac, bytes, s);
    switch (c.logN) {
        case 10: launch_rows_mac<10>(c, d_jobs, njobs, s); break;
        case 11: launch_rows_mac<11>(c, d_jobs, njobs, s); break;
        case 12: launch_rows_mac<12>(c, d_jobs, njobs, s); break;
        case 13: launch_rows_mac<13>(c, d_jobs, njobs, s); break;
        case 14: launch_rows_mac<14>(c, d_jobs, njobs, s); break;
        case 15: launch_rows_mac<15>(c, d_jobs, njobs, s); break;
        case 16: launch_rows_mac<16>(c, d_jobs, njobs, s); break;
        default: fail(kInvalid, "ntt: ring degree must be 2^10 .. 2^16");
    }
    check_cuda(cudaGetLastError(), "key inner product launch");
}

void ntt_rows_epilogue_jobs(const Context& c, const NttEpiJob* d_jobs, int njobs, double bytes, cudaStream_t s) {
    if (njobs <= 0) return;
    // booked as NTT work: the phase's share plus the epilogue's words (ntt_epilogue_bytes)
    Probe probe(kClsNtt, bytes, s);
    // 8 residues per thread with twiddles from the table whatever the tuner chose for the plain
    // row phase: the prefetched operands take 32 KiB of shared memory, which leaves 4 blocks per
    // SM only in this geometry
    switch (c.logN) {
        case 10: launch_rows_epi<10, 3, false>(c, d_jobs, njobs, s); break;
        case 11: launch_rows_epi<11, 3, false>(c, d_jobs, njobs, s); break;
        case 12: launch_rows_epi<12, 3, false>(c, d_jobs, njobs, s); break;
        case 13: launch_rows_epi<13, 3, false>(c, d_jobs, njobs, s); break;
        case 14: launch_rows_epi<14, 3, false>(c, d_jobs, njobs, s); break;
        case 15: launch_rows_epi<15, 3, false>(c, d_jobs, njobs, s); break;
        case 16: launch_rows_epi<16, 3, false>(c, d_jobs, njobs, s); break;
        default: fail(kInvalid, "ntt: ring degree must be 2^10 .. 2^16");
    }
    check_cuda(cudaGetLastError(), "ntt epilogue launch");
}

// Time every geometry of every (direction, phase) the way the batched circuits launch the
// transform: job-table launches of 64 limbs over a scratch batch larger than the L2 cache (160 MB
// of limbs) cycling over the context's moduli, so lazy and full-reduction moduli are both
// represented; best of three passes after one warm-up.  A geometry replaces the default
// (8 residues per thread, staged twiddles) only when it is at least 5 % faster, so timing noise
// does not flip the choice.  Phases are timed on their own: each is one full pass over the
// batch whatever the other phase does, and every geometry computes the same words, so the
// choices combine freely.
void ntt_autotune(Context& c) {
    {
        std::lock_guard<std::mutex> g(g_tune_mutex);
        auto it = g_tuned.find(tune_key(c));
        if (it != g_tuned.end()) {
            c.tuning = it->second;
            take_tuning(c);
            return;
        }
    }
    const size_t N = c.N;
    const int kTuneLimbs = (int)((size_t{160} << 20) / (8 * N));
    const int kTuneBatch = 64;
    const int nm = (int)(c.nq + c.np);
    check_cuda(cudaSetDevice(c.device), "cudaSetDevice");
    uint64_t* buf = nullptr;
    NttJob* d_jobs = nullptr;
    if (cudaMalloc(&buf, (size_t)kTuneLimbs * N * 8) != cudaSuccess ||
        cudaMalloc(&d_jobs, (size_t)kTuneLimbs * sizeof(NttJob)) != cudaSuccess) {
        // no room for the timing batch: keep the default geometry (tuning.limbs = 0 says so)
        cudaGetLastError();
        cudaFree(buf);
        return;
    }
    try {
        c.rows16(true);
    } catch (const Error&) {
        cudaFree(buf);
        cudaFree(d_jobs);
        return;
    }
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    NttTuning tn{};
    auto release = [&] {
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (s) cudaStreamDestroy(s);
        cudaFree(buf);
        cudaFree(d_jobs);
    };
    try {
        check_cuda(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "ntt autotune: stream");
        check_cuda(cudaEventCreate(&e0), "ntt autotune: event");
        check_cuda(cudaEventCreate(&e1), "ntt autotune: event");
        check_cuda(cudaMemsetAsync(buf, 0, (size_t)kTuneLimbs * N * 8, s), "ntt autotune: clear");
        std::vector<NttJob> jobs(kTuneLimbs);
        for (int l = 0; l < kTuneLimbs; ++l) jobs[l] = {buf + (size_t)l * N, buf + (size_t)l * N, l % nm, 0};
        check_cuda(cudaMemcpyAsync(d_jobs, jobs.data(), jobs.size() * sizeof(NttJob), cudaMemcpyHostToDevice, s),
                   "ntt autotune: jobs");
        for (int d = 0; d < 2; ++d)
            for (int p = 0; p < 2; ++p) {
                for (int v = 0; v < kNttGeometries; ++v) {
                    float t_best = 1e30f;
                    for (int rep = 0; rep < 4; ++rep) {
                        check_cuda(cudaEventRecord(e0, s), "ntt autotune: record");
                        // launches of kTuneBatch limbs, the size of a batched key switch's NTT
                        // launch, so block tails and occupancy weigh as they do in the circuits
                        for (int l0 = 0; l0 < kTuneLimbs; l0 += kTuneBatch)
                            phase_dispatch(c, d == 0, p == 1, v, nullptr, 0, 0, 0, LimbMap{0, 0, 0}, d_jobs + l0,
                                           std::min(kTuneBatch, kTuneLimbs - l0), s);
                        check_cuda(cudaEventRecord(e1, s), "ntt autotune: record");
                        check_cuda(cudaEventSynchronize(e1), "ntt autotune: wait");
                        float ms = 0;
                        check_cuda(cudaEventElapsedTime(&ms, e0, e1), "ntt autotune: time");
                        if (rep > 0) t_best = std::min(t_best, ms);
                    }
                    tn.ms[d][p][v] = t_best;
                }
                int best_v = 0;
                for (int v = 1; v < kNttGeometries; ++v)
                    if (tn.ms[d][p][v] < 0.95f * tn.ms[d][p][0] && tn.ms[d][p][v] < tn.ms[d][p][best_v]) best_v = v;
                tn.chosen[d][p] = best_v;
            }
        tn.limbs = kTuneLimbs;
    } catch (...) {
        release();
        throw;
    }
    release();
    c.tuning = tn;
    take_tuning(c);
    std::lock_guard<std::mutex> g(g_tune_mutex);
    g_tuned[tune_key(c)] = tn;
}

}  // namespace wg
