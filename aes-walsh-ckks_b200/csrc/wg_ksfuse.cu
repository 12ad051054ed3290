// Key-switch ModUp and ModDown, and the rescale's remainder step, fused with the NTT column
// phases around them.
//
// Unfused, a hybrid key switch (ckks_hybrid_key_switch_inplace,
// src/ckks/operations/keyswitch/ckks_keyswitch.cpp:1330-1641) moves every intermediate limb
// through device memory between separate launches: the inverse NTT of the key term writes its
// coefficients, ModUp reads them and writes the digits, the forward NTT reads and rewrites the
// digits twice (one pass per phase); after the key inner product the same happens around
// ModDown.  Here one CTA per (digit or accumulator, column tile) runs
//
//   inverse column phase of its source limbs -> N^-1 -> ModUp / ModDown -> forward column
//   phase of every output limb
//
// in shared memory (wg_ksfuse.cuh), so the coefficient-form source limbs and the un-transformed
// outputs never reach device memory.  Per switch at walsh15's top level (L = 13, K = 4, three
// digits of 5, 5 and 3 source limbs, 38 destination limbs) the NTT/ModUp/ModDown traffic falls
// from 425 to 255 limb passes of 8N bytes, with the same words written.  Launches too small to fill
// the device divide a job's output limbs over several CTAs (split_of).
#include <algorithm>
#include <utility>

#include "wg_internal.hpp"
#include "wg_ksfuse.cuh"

namespace wg {
namespace {
using namespace ksf;
using ntt::TwPair;

// The column rounds on a thread's elements, exchanged through `sm` (which others may still read on
// entry).
template <class G, bool FWD, int RD, class Arith>
__device__ __forceinline__ void col_round(uint64_t* sm, typename Arith::V* v, int tile, int t, const Arith& ar,
                                          const TwPair* tw) {
    using R = ntt::Round<G::LOG, FWD, true, G::BITS, false, RD, kTile>;
    const int sub = R::P::sub_of(t), o = R::P::o_of(t);
    if constexpr (RD > 0) {
        __syncthreads();
        ntt::Round<G::LOG, FWD, true, G::BITS, false, RD - 1, kTile>::template scatter<Arith>(sm, sub, o, v);
        __syncthreads();
        R::template gather<Arith>(sm, sub, o, v);
    }
    R::stages(v, sub, o, tile, ar, tw);
}
template <class G, bool FWD, class Arith, int... RD>
__device__ __forceinline__ void col_rounds(std::integer_sequence<int, RD...>, uint64_t* sm, typename Arith::V* v, int tile,
                                           int t, const Arith& ar, const TwPair* tw) {
    (col_round<G, FWD, RD>(sm, v, tile, t, ar, tw), ...);
}
template <class G, bool FWD, class Arith>
__device__ __forceinline__ void columns(uint64_t* sm, typename Arith::V* v, int tile, int t, const Arith& ar,
                                        const TwPair* tw) {
    col_rounds<G, FWD>(std::make_integer_sequence<int, G::ROUNDS>{}, sm, v, tile, t, ar, tw);
}

// The inverse column phase of thread t's slots of one source limb: `scale` turns the rounds' values
// (doubles or words) into the canonical ones kept there.
template <class G, class ScaleFp, class ScaleWords>
__device__ __forceinline__ void inverse_slots(uint64_t* sm, uint64_t* slots, int tile, int t, const Modulus& m,
                                              const TwPair* tw, ScaleFp scale_f, ScaleWords scale_w) {
    if (m.q < fp::kLimit) {
        double v[G::E];
#pragma unroll
        for (int k = 0; k < G::E; ++k) v[k] = fp::bits_double(slots[k * G::THREADS + t]);
        columns<G, false>(sm, v, tile, t, ntt::fp_arith(m), tw);
        scale_f(v);
#pragma unroll
        for (int k = 0; k < G::E; ++k) slots[k * G::THREADS + t] = fp::double_bits(v[k]);
    } else {
        uint64_t v[G::E];
#pragma unroll
        for (int k = 0; k < G::E; ++k) v[k] = slots[k * G::THREADS + t];
        columns<G, false>(sm, v, tile, t, ntt::WordArith<false>{m.q}, tw);
        scale_w(v);
#pragma unroll
        for (int k = 0; k < G::E; ++k) slots[k * G::THREADS + t] = v[k];
    }
}

// The forward column phase of one output limb from thread t's coefficients: value_f fills doubles
// (unreduced), value_w canonical words.
template <class G, class ValueFp, class ValueWords>
__device__ __forceinline__ void forward_limb(uint64_t* sm, uint64_t* limb, int tile, int t, const Modulus& m,
                                             const TwPair* tw, ValueFp value_f, ValueWords value_w) {
    using End = typename G::template FwdRound<G::ROUNDS - 1>;
    uint64_t w[G::E];
    if (m.q < fp::kLimit) {
        double v[G::E];
        value_f(v);
        columns<G, true>(sm, v, tile, t, ntt::fp_arith(m), tw);
#pragma unroll
        for (int k = 0; k < G::E; ++k) w[k] = fp::double_bits(v[k]);
    } else {
        value_w(w);
        // moduli below kLazyForwardLimit skip the per-butterfly reduction, as k_ntt_phase does
        if (m.q < ntt::kLazyForwardLimit)
            columns<G, true>(sm, w, tile, t, ntt::WordArith<true>{m.q}, tw);
        else
            columns<G, true>(sm, w, tile, t, ntt::WordArith<false>{m.q}, tw);
    }
    store_limb<End>(w, limb, tile, t);
}

// Shared memory: the sources' slots (TILE words each), then the exchange tile.  Four blocks an SM: up to
// five sources (50 KB) leave room for them, and four residues a thread take 64 registers, eight 128 (with
// more sources fewer blocks fit, and split_of, which counts four, divides a small launch further than one
// wave).  A rescale has one source and takes 80 registers.
constexpr int kResident = 4;
constexpr int kRescaleResident = 6;
template <class G>
constexpr size_t fused_smem(int sources) {
    return 8 * ((size_t)G::TILE * sources + G::PAD);
}

// Blocks per job and column tile: a job's output limbs are divided over `split` blocks, each of which
// repeats the source limbs' inverse column phase.  A launch that fills the device takes one; smaller
// launches (one or a few ciphertexts) take as many as the device has room for, up to the point where
// a block's outputs are half its sources: the repeated work then costs more than the shorter chain of
// a block saves.
int split_of(const Context& c, int njobs, int tiles, int resident, int sources, int outputs) {
    const int room = resident * c.sm_count / std::max(1, njobs * tiles);
    const int most = (2 * outputs + sources - 1) / std::max(1, sources);
    return std::max(1, std::min({room, most, outputs}));
}
template <class G>
__device__ __forceinline__ Share block_share() {
    return share_of(blockIdx.x, gridDim.x, G::TILES);
}

// Block (tile and share of the outputs, job): one digit's column tile.
template <class G>
__global__ void __launch_bounds__(G::THREADS, kResident)
    k_modup_ntt(const ModUpNttJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods,
                const TwPair* __restrict__ tw_base) {
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const ModUpNttJob job = jobs[j];
    const ModUpDesc& d = *job.desc;
    const int n = d.src_count, first = d.src_first;
    const Share sh = block_share<G>();
    if (sh.begin >= d.dst_count) return;
    const int tile = sh.tile, t = threadIdx.x;
    uint64_t* work = smem + n * G::TILE;

    // every source limb in flight at once, each awaited just before its inverse column phase
    for (int i = 0; i < n; ++i) {
        load_slots_async<G>(smem + i * G::TILE, job.src + (size_t)(first + i) * G::N, tile, t);
        cp_async_commit();
    }
    SourceKinds kinds;
    double alpha[G::E];
#pragma unroll
    for (int k = 0; k < G::E; ++k) alpha[k] = 0.0;
    for (int i = 0; i < n; ++i) {
        const int mi = first + i;
        const Modulus m = mods[mi];
        kinds.set(i, m.q);
        cp_async_wait_upto(n - 1 - i);
        inverse_slots<G>(
            work, smem + i * G::TILE, tile, t, m, tw_base + (size_t)mi * 2 * G::N + G::N,
            [&](double* v) { modup_scale_fp<G>(v, d, i, m.qd, alpha); },
            [&](uint64_t* v) {
                scale_n_inv<G::E>(v, m);
                modup_scale<G>(v, d, i, m.q, alpha);
            });
    }
    uint32_t hps[G::E];
#pragma unroll
    for (int k = 0; k < G::E; ++k) hps[k] = hps_count(alpha[k], n);
    for (int dst = sh.begin; dst < d.dst_count; dst += sh.step) {
        const int mi = __ldg(d.dst_mod + dst);
        const Modulus m = mods[mi];
        forward_limb<G>(
            work, job.digit + (size_t)__ldg(d.dst_limb + dst) * G::N, tile, t, m, tw_base + (size_t)mi * 2 * G::N,
            [&](double* v) { modup_value_fp<G>(v, smem, t, d, dst, m, hps, kinds); },
            [&](uint64_t* v) { modup_value<G>(v, smem, t, d, dst, m.q, hps, kinds.fp64); });
    }
}

// Block (tile and share, job): one accumulator polynomial's column tile.  FMA: the alpha sum's rounding
// (moddown_hps).
template <class G, bool FMA>
__global__ void __launch_bounds__(G::THREADS, kResident)
    k_moddown_ntt(const ModDownNttJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods, int nq, int K,
                  const TwPair* __restrict__ tw_base) {
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const ModDownNttJob job = jobs[j];
    const Share sh = block_share<G>();
    if (sh.begin >= job.L) return;
    const int tile = sh.tile, t = threadIdx.x;
    uint64_t* work = smem + K * G::TILE;
    const Modulus* pmods = mods + nq;

    for (int pi = 0; pi < K; ++pi) {
        load_slots_async<G>(smem + pi * G::TILE, job.src_p + (size_t)pi * G::N, tile, t);
        cp_async_commit();
    }
    SourceKinds kinds;
    for (int pi = 0; pi < K; ++pi) {
        const Modulus m = pmods[pi];
        kinds.set(pi, m.q);
        cp_async_wait_upto(K - 1 - pi);
        inverse_slots<G>(
            work, smem + pi * G::TILE, tile, t, m, tw_base + (size_t)(nq + pi) * 2 * G::N + G::N,
            [&](double* v) { scale_fp<G::E>(v, m.n_inv_w, m.n_inv_wq, m.qd); }, [&](uint64_t* v) { scale_n_inv<G::E>(v, m); });
    }
    uint32_t hps[G::E];
    moddown_hps<G, FMA>(smem, t, pmods, K, hps, kinds.fp64);
    for (int qi = sh.begin; qi < job.L; qi += sh.step) {
        const Modulus m = mods[qi];
        const uint64_t *iv = job.inv + (size_t)qi * K, *ivs = job.inv_s + (size_t)qi * K;
        forward_limb<G>(
            work, job.out + (size_t)qi * G::N, tile, t, m, tw_base + (size_t)qi * 2 * G::N,
            [&](double* v) {
                moddown_value_fp<G>(v, smem, t, K, m, iv, ivs, job.inv_fp + (size_t)qi * K, hps, kinds);
            },
            [&](uint64_t* v) { moddown_value<G>(v, smem, t, K, m.q, iv, ivs, hps, kinds.fp64); });
    }
}

// Block (tile and share, job): one polynomial's column tile of a rescale.
template <class G>
__global__ void __launch_bounds__(G::THREADS, kRescaleResident)
    k_rescale_ntt(const RescaleNttJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods,
                  const TwPair* __restrict__ tw_base) {
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const RescaleNttJob job = jobs[j];
    const int t = threadIdx.x, lv = job.lv;
    const Share sh = block_share<G>();
    if (sh.begin >= lv) return;
    const int tile = sh.tile;
    uint64_t* drop = smem;
    uint64_t* work = smem + G::TILE;
    const Modulus mp = mods[lv];
    const bool fp_drop = mp.q < fp::kLimit;
    uint64_t w[G::E];
    load_limb<typename G::template InvRound<0>>(w, job.drop, tile, t);
#pragma unroll
    for (int k = 0; k < G::E; ++k)  // lazily reduced words of an FP64 limb: below 2 q
        drop[k * G::THREADS + t] = fp_drop && job.words ? fp::double_bits(fp::from_word(w[k])) : w[k];
    inverse_slots<G>(
        work, drop, tile, t, mp, tw_base + (size_t)lv * 2 * G::N + G::N,
        [&](double* v) { scale_fp<G::E>(v, mp.n_inv_w, mp.n_inv_wq, mp.qd); }, [&](uint64_t* v) { scale_n_inv<G::E>(v, mp); });
    if (job.keep && sh.begin == 0) {
#pragma unroll
        for (int k = 0; k < G::E; ++k) w[k] = slot_word(drop[k * G::THREADS + t], fp_drop);
        store_limb<typename G::template InvRound<G::ROUNDS - 1>>(w, job.keep, tile, t);
    }
    for (int qi = sh.begin; qi < lv; qi += sh.step) {
        const Modulus m = mods[qi];
        const uint64_t one_s = __ldg(job.rc + qi), half = __ldg(job.rc + 3 * lv + qi);
        forward_limb<G>(
            work, job.rem + (size_t)qi * G::N, tile, t, m, tw_base + (size_t)qi * 2 * G::N,
            [&](double* v) { rescale_value_fp<G>(v, drop, t, mp.q, m, one_s, half, fp_drop); },
            [&](uint64_t* v) { rescale_value<G>(v, drop, t, mp.q, m.q, one_s, half, fp_drop); });
    }
}

template <int LOGN>
void launch_rescale(const Context& c, const RescaleNttJob* jobs, int njobs, int max_out, cudaStream_t s) {
    using G = Geom<LOGN, kRescaleBits>;
    const dim3 grid(G::TILES * split_of(c, njobs, G::TILES, kRescaleResident, 1, max_out), njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_rescale_ntt<G><<<grid, G::THREADS, fused_smem<G>(1), s>>>(jobs, njobs, c.d_mod,
                                                                      c.twiddles(3));
}

template <class G>
void launch_modup_g(const Context& c, const ModUpNttJob* jobs, int njobs, int max_src, int max_out, cudaStream_t s) {
    allow_shared<k_modup_ntt<G>>(c.device, fused_smem<G>(kMaxDigitWidth));
    const dim3 grid(G::TILES * split_of(c, njobs, G::TILES, kResident, max_src, max_out),
                    njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_modup_ntt<G><<<grid, G::THREADS, fused_smem<G>(max_src), s>>>(jobs, njobs, c.d_mod, c.twiddles(3));
}

template <int LOGN>
void launch_modup(const Context& c, const ModUpNttJob* jobs, int njobs, int max_src, int max_out, cudaStream_t s) {
    if (c.word_moduli)
        launch_modup_g<Geom<LOGN, kModUpBits>>(c, jobs, njobs, max_src, max_out, s);
    else
        launch_modup_g<Geom<LOGN, kModUpFpBits>>(c, jobs, njobs, max_src, max_out, s);
}

template <int LOGN, bool FMA>
void launch_moddown_f(const Context& c, const ModDownNttJob* jobs, int njobs, int max_out, cudaStream_t s) {
    using G = Geom<LOGN, kModDownBits>;
    allow_shared<k_moddown_ntt<G, FMA>>(c.device, fused_smem<G>(kMaxPLimbs));
    const dim3 grid(G::TILES * split_of(c, njobs, G::TILES, kResident, (int)c.np, max_out),
                    njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_moddown_ntt<G, FMA><<<grid, G::THREADS, fused_smem<G>((int)c.np), s>>>(
        jobs, njobs, c.d_mod, (int)c.nq, (int)c.np, c.twiddles(3));
}

template <int LOGN>
void launch_moddown(const Context& c, const ModDownNttJob* jobs, int njobs, int max_out, bool fma, cudaStream_t s) {
    if (fma)
        launch_moddown_f<LOGN, true>(c, jobs, njobs, max_out, s);
    else
        launch_moddown_f<LOGN, false>(c, jobs, njobs, max_out, s);
}

}  // namespace

void modup_ntt_jobs(const Context& c, const ModUpNttJob* d_jobs, int njobs, int max_src, int max_out, double bytes,
                    cudaStream_t s) {
    if (njobs <= 0) return;
    if (max_src < 1 || max_src > kMaxDigitWidth) fail(kInvalid, "fused modup: digit width out of range");
    Probe probe(kClsModUp, bytes, s);
    switch (c.logN) {
        case 10: launch_modup<10>(c, d_jobs, njobs, max_src, max_out, s); break;
        case 11: launch_modup<11>(c, d_jobs, njobs, max_src, max_out, s); break;
        case 12: launch_modup<12>(c, d_jobs, njobs, max_src, max_out, s); break;
        case 13: launch_modup<13>(c, d_jobs, njobs, max_src, max_out, s); break;
        case 14: launch_modup<14>(c, d_jobs, njobs, max_src, max_out, s); break;
        case 15: launch_modup<15>(c, d_jobs, njobs, max_src, max_out, s); break;
        case 16: launch_modup<16>(c, d_jobs, njobs, max_src, max_out, s); break;
        default: fail(kInvalid, "fused modup: ring degree must be 2^10 .. 2^16");
    }
    check_cuda(cudaGetLastError(), "fused modup launch");
}

void rescale_ntt_jobs(const Context& c, const RescaleNttJob* d_jobs, int njobs, int max_out, double bytes,
                      cudaStream_t s) {
    if (njobs <= 0) return;
    Probe probe(kClsElementwise, bytes, s);
    switch (c.logN) {
        case 10: launch_rescale<10>(c, d_jobs, njobs, max_out, s); break;
        case 11: launch_rescale<11>(c, d_jobs, njobs, max_out, s); break;
        case 12: launch_rescale<12>(c, d_jobs, njobs, max_out, s); break;
        case 13: launch_rescale<13>(c, d_jobs, njobs, max_out, s); break;
        case 14: launch_rescale<14>(c, d_jobs, njobs, max_out, s); break;
        case 15: launch_rescale<15>(c, d_jobs, njobs, max_out, s); break;
        case 16: launch_rescale<16>(c, d_jobs, njobs, max_out, s); break;
        default: fail(kInvalid, "fused rescale: ring degree must be 2^10 .. 2^16");
    }
    check_cuda(cudaGetLastError(), "fused rescale launch");
}

void moddown_ntt_jobs(const Context& c, const ModDownNttJob* d_jobs, int njobs, int max_out, double bytes,
                      cudaStream_t s, bool fma_alpha) {
    if (njobs <= 0) return;
    if (c.np < 1 || c.np > (size_t)kMaxPLimbs) fail(kInvalid, "fused moddown: P limb count out of range");
    Probe probe(kClsModDown, bytes, s);
    switch (c.logN) {
        case 10: launch_moddown<10>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        case 11: launch_moddown<11>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        case 12: launch_moddown<12>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        case 13: launch_moddown<13>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        case 14: launch_moddown<14>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        case 15: launch_moddown<15>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        case 16: launch_moddown<16>(c, d_jobs, njobs, max_out, fma_alpha, s); break;
        default: fail(kInvalid, "fused moddown: ring degree must be 2^10 .. 2^16");
    }
    check_cuda(cudaGetLastError(), "fused moddown launch");
}

}  // namespace wg
