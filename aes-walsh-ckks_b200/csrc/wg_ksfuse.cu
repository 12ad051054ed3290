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
template <int LOGN, bool FWD, int RD, class Arith>
__device__ __forceinline__ void col_round(uint64_t* sm, typename Arith::V* v, int tile, int t, const Arith& ar,
                                          const TwPair* tw) {
    using R = ntt::Round<LOGN, FWD, true, 3, false, RD, kTile>;
    const int sub = R::P::sub_of(t), o = R::P::o_of(t);
    if constexpr (RD > 0) {
        __syncthreads();
        ntt::Round<LOGN, FWD, true, 3, false, RD - 1, kTile>::template scatter<Arith>(sm, sub, o, v);
        __syncthreads();
        R::template gather<Arith>(sm, sub, o, v);
    }
    R::stages(v, sub, o, tile, ar, tw);
}
template <int LOGN, bool FWD, class Arith, int... RD>
__device__ __forceinline__ void col_rounds(std::integer_sequence<int, RD...>, uint64_t* sm, typename Arith::V* v, int tile,
                                           int t, const Arith& ar, const TwPair* tw) {
    (col_round<LOGN, FWD, RD>(sm, v, tile, t, ar, tw), ...);
}
template <int LOGN, bool FWD, class Arith>
__device__ __forceinline__ void columns(uint64_t* sm, typename Arith::V* v, int tile, int t, const Arith& ar,
                                        const TwPair* tw) {
    col_rounds<LOGN, FWD>(std::make_integer_sequence<int, Geom<LOGN>::ROUNDS>{}, sm, v, tile, t, ar, tw);
}

// The inverse column phase of thread t's slots of one source limb: `scale` turns the rounds' values
// (doubles or words) into the canonical ones kept there.
template <int LOGN, class ScaleFp, class ScaleWords>
__device__ __forceinline__ void inverse_slots(uint64_t* sm, uint64_t* slots, int tile, int t, const Modulus& m,
                                              const TwPair* tw, ScaleFp scale_f, ScaleWords scale_w) {
    using G = Geom<LOGN>;
    if (m.q < fp::kLimit) {
        double v[G::E];
#pragma unroll
        for (int k = 0; k < G::E; ++k) v[k] = fp::bits_double(slots[k * G::THREADS + t]);
        columns<LOGN, false>(sm, v, tile, t, ntt::fp_arith(m), tw);
        scale_f(v);
#pragma unroll
        for (int k = 0; k < G::E; ++k) slots[k * G::THREADS + t] = fp::double_bits(v[k]);
    } else {
        uint64_t v[G::E];
#pragma unroll
        for (int k = 0; k < G::E; ++k) v[k] = slots[k * G::THREADS + t];
        columns<LOGN, false>(sm, v, tile, t, ntt::WordArith<false>{m.q}, tw);
        scale_w(v);
#pragma unroll
        for (int k = 0; k < G::E; ++k) slots[k * G::THREADS + t] = v[k];
    }
}

// The forward column phase of one output limb from thread t's coefficients: value_f fills doubles
// (unreduced), value_w canonical words.
template <int LOGN, class ValueFp, class ValueWords>
__device__ __forceinline__ void forward_limb(uint64_t* sm, uint64_t* limb, int tile, int t, const Modulus& m,
                                             const TwPair* tw, ValueFp value_f, ValueWords value_w) {
    using G = Geom<LOGN>;
    using End = typename G::template FwdRound<G::ROUNDS - 1>;
    uint64_t w[G::E];
    if (m.q < fp::kLimit) {
        double v[G::E];
        value_f(v);
        columns<LOGN, true>(sm, v, tile, t, ntt::fp_arith(m), tw);
#pragma unroll
        for (int k = 0; k < G::E; ++k) w[k] = fp::double_bits(v[k]);
    } else {
        value_w(w);
        // moduli below kLazyForwardLimit skip the per-butterfly reduction, as k_ntt_phase does
        if (m.q < ntt::kLazyForwardLimit)
            columns<LOGN, true>(sm, w, tile, t, ntt::WordArith<true>{m.q}, tw);
        else
            columns<LOGN, true>(sm, w, tile, t, ntt::WordArith<false>{m.q}, tw);
    }
    store_limb<End>(w, limb, tile, t);
}

// Shared memory: the sources' slots (TILE words each), then the exchange tile.  Resident blocks per SM
// (the launch bounds) follow from it: up to 4 sources of 8 KiB leave room for 5 blocks, the
// rescale's single one for 6 (register-limited).
template <int LOGN>
constexpr size_t fused_smem(int sources) {
    return 8 * ((size_t)Geom<LOGN>::TILE * sources + Geom<LOGN>::PAD);
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
// The outputs [begin, end) of a block: gridDim.x = TILES * split.
struct Share {
    int tile, begin, end;
};
template <int LOGN>
__device__ __forceinline__ Share block_share(int outputs) {
    constexpr int tiles = Geom<LOGN>::TILES;
    const int split = gridDim.x / tiles, part = blockIdx.x / tiles;
    const int chunk = (outputs + split - 1) / split;
    const int begin = part * chunk;
    return {(int)(blockIdx.x % tiles), begin, begin + chunk < outputs ? begin + chunk : outputs};
}

// Block (tile and share of the outputs, job): one digit's column tile.  W >= every job's digit width.
template <int LOGN, int W>
__global__ void __launch_bounds__(Geom<LOGN>::THREADS, W <= 4 ? 5 : 4)
    k_modup_ntt(const ModUpNttJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods,
                const TwPair* __restrict__ tw_base) {
    using G = Geom<LOGN>;
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const ModUpNttJob job = jobs[j];
    const ModUpDesc& d = *job.desc;
    const int n = d.src_count, first = d.src_first;
    const Share sh = block_share<LOGN>(d.dst_count);
    if (sh.begin >= sh.end) return;
    const int tile = sh.tile, t = threadIdx.x;
    uint64_t* work = smem + n * G::TILE;

    // every source limb in flight at once, each awaited just before its inverse column phase
    for (int i = 0; i < n; ++i) {
        load_slots_async<LOGN>(smem + i * G::TILE, job.src + (size_t)(first + i) * G::N, tile, t);
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
        inverse_slots<LOGN>(
            work, smem + i * G::TILE, tile, t, m, tw_base + (size_t)mi * 2 * G::N + G::N,
            [&](double* v) { modup_scale_fp(v, d, i, m.qd, alpha); },
            [&](uint64_t* v) {
                scale_n_inv(v, m);
                modup_scale(v, d, i, m.q, alpha);
            });
    }
    uint32_t hps[G::E];
#pragma unroll
    for (int k = 0; k < G::E; ++k) hps[k] = hps_count(alpha[k], n);
    for (int dst = sh.begin; dst < sh.end; ++dst) {
        const int mi = __ldg(d.dst_mod + dst);
        const Modulus m = mods[mi];
        forward_limb<LOGN>(
            work, job.digit + (size_t)__ldg(d.dst_limb + dst) * G::N, tile, t, m, tw_base + (size_t)mi * 2 * G::N,
            [&](double* v) { modup_value_fp<LOGN>(v, smem, t, d, dst, m, hps, kinds); },
            [&](uint64_t* v) { modup_value<LOGN, W>(v, smem, t, d, dst, m.q, hps, kinds.fp64); });
    }
}

// Block (tile and share, job): one accumulator polynomial's column tile.  FMA: the alpha sum's rounding
// (moddown_hps); KW >= K.
template <int LOGN, bool FMA, int KW>
__global__ void __launch_bounds__(Geom<LOGN>::THREADS, KW <= 4 ? 5 : 4)
    k_moddown_ntt(const ModDownNttJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods, int nq, int K,
                  const TwPair* __restrict__ tw_base) {
    using G = Geom<LOGN>;
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const ModDownNttJob job = jobs[j];
    const Share sh = block_share<LOGN>(job.L);
    if (sh.begin >= sh.end) return;
    const int tile = sh.tile, t = threadIdx.x;
    uint64_t* work = smem + K * G::TILE;
    const Modulus* pmods = mods + nq;

    for (int pi = 0; pi < K; ++pi) {
        load_slots_async<LOGN>(smem + pi * G::TILE, job.src_p + (size_t)pi * G::N, tile, t);
        cp_async_commit();
    }
    SourceKinds kinds;
    for (int pi = 0; pi < K; ++pi) {
        const Modulus m = pmods[pi];
        kinds.set(pi, m.q);
        cp_async_wait_upto(K - 1 - pi);
        inverse_slots<LOGN>(
            work, smem + pi * G::TILE, tile, t, m, tw_base + (size_t)(nq + pi) * 2 * G::N + G::N,
            [&](double* v) { scale_fp(v, m.n_inv_w, m.n_inv_wq, m.qd); }, [&](uint64_t* v) { scale_n_inv(v, m); });
    }
    uint32_t hps[G::E];
    moddown_hps<LOGN, KW, FMA>(smem, t, pmods, K, hps, kinds.fp64);
    for (int qi = sh.begin; qi < sh.end; ++qi) {
        const Modulus m = mods[qi];
        const uint64_t *iv = job.inv + (size_t)qi * K, *ivs = job.inv_s + (size_t)qi * K;
        forward_limb<LOGN>(
            work, job.out + (size_t)qi * G::N, tile, t, m, tw_base + (size_t)qi * 2 * G::N,
            [&](double* v) {
                moddown_value_fp<LOGN>(v, smem, t, K, m, iv, ivs, job.inv_fp + (size_t)qi * K, hps, kinds);
            },
            [&](uint64_t* v) { moddown_value<LOGN, KW>(v, smem, t, K, m.q, iv, ivs, hps, kinds.fp64); });
    }
}

// Block (tile and share, job): one polynomial's column tile of a rescale.
template <int LOGN>
__global__ void __launch_bounds__(Geom<LOGN>::THREADS, 6)
    k_rescale_ntt(const RescaleNttJob* __restrict__ jobs, int njobs, const Modulus* __restrict__ mods,
                  const TwPair* __restrict__ tw_base) {
    using G = Geom<LOGN>;
    const int j = blockIdx.y + 65535 * blockIdx.z;
    if (j >= njobs) return;
    extern __shared__ __align__(16) uint64_t smem[];
    const RescaleNttJob job = jobs[j];
    const int t = threadIdx.x, lv = job.lv;
    const Share sh = block_share<LOGN>(lv);
    if (sh.begin >= sh.end) return;
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
    inverse_slots<LOGN>(
        work, drop, tile, t, mp, tw_base + (size_t)lv * 2 * G::N + G::N,
        [&](double* v) { scale_fp(v, mp.n_inv_w, mp.n_inv_wq, mp.qd); }, [&](uint64_t* v) { scale_n_inv(v, mp); });
    if (job.keep && sh.begin == 0) {
#pragma unroll
        for (int k = 0; k < G::E; ++k) w[k] = slot_word(drop[k * G::THREADS + t], fp_drop);
        store_limb<typename G::template InvRound<G::ROUNDS - 1>>(w, job.keep, tile, t);
    }
    for (int qi = sh.begin; qi < sh.end; ++qi) {
        const Modulus m = mods[qi];
        const uint64_t one_s = __ldg(job.rc + qi), half = __ldg(job.rc + 3 * lv + qi);
        forward_limb<LOGN>(
            work, job.rem + (size_t)qi * G::N, tile, t, m, tw_base + (size_t)qi * 2 * G::N,
            [&](double* v) { rescale_value_fp<LOGN>(v, drop, t, mp.q, m, one_s, half, fp_drop); },
            [&](uint64_t* v) { rescale_value<LOGN>(v, drop, t, mp.q, m.q, one_s, half, fp_drop); });
    }
}

template <int LOGN>
void launch_rescale(const Context& c, const RescaleNttJob* jobs, int njobs, int max_out, cudaStream_t s) {
    using G = Geom<LOGN>;
    const dim3 grid(G::TILES * split_of(c, njobs, G::TILES, 6, 1, max_out), njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_rescale_ntt<LOGN><<<grid, G::THREADS, fused_smem<LOGN>(1), s>>>(jobs, njobs, c.d_mod,
                                                                      c.twiddles(3));
}

template <int LOGN, int W>
void launch_modup_w(const Context& c, const ModUpNttJob* jobs, int njobs, int max_src, int max_out, cudaStream_t s) {
    using G = Geom<LOGN>;
    static const bool opted = [] {
        cudaFuncSetAttribute(k_modup_ntt<LOGN, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)fused_smem<LOGN>(W));
        return true;
    }();
    (void)opted;
    const dim3 grid(G::TILES * split_of(c, njobs, G::TILES, W <= 4 ? 5 : 4, max_src, max_out),
                    njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_modup_ntt<LOGN, W><<<grid, G::THREADS, fused_smem<LOGN>(max_src), s>>>(jobs, njobs, c.d_mod,
                                                                              c.twiddles(3));
}

template <int LOGN>
void launch_modup(const Context& c, const ModUpNttJob* jobs, int njobs, int max_src, int max_out, cudaStream_t s) {
    if (max_src <= 4)
        launch_modup_w<LOGN, 4>(c, jobs, njobs, max_src, max_out, s);
    else if (max_src <= 8)
        launch_modup_w<LOGN, 8>(c, jobs, njobs, max_src, max_out, s);
    else
        launch_modup_w<LOGN, kMaxDigitWidth>(c, jobs, njobs, max_src, max_out, s);
}

template <int LOGN, bool FMA, int KW>
void launch_moddown_k(const Context& c, const ModDownNttJob* jobs, int njobs, int max_out, cudaStream_t s) {
    using G = Geom<LOGN>;
    static const bool opted = [] {
        cudaFuncSetAttribute(k_moddown_ntt<LOGN, FMA, KW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)fused_smem<LOGN>(KW));
        return true;
    }();
    (void)opted;
    const dim3 grid(G::TILES * split_of(c, njobs, G::TILES, KW <= 4 ? 5 : 4, (int)c.np, max_out),
                    njobs < 65535 ? njobs : 65535, (njobs + 65534) / 65535);
    k_moddown_ntt<LOGN, FMA, KW><<<grid, G::THREADS, fused_smem<LOGN>((int)c.np), s>>>(
        jobs, njobs, c.d_mod, (int)c.nq, (int)c.np, c.twiddles(3));
}

template <int LOGN, bool FMA>
void launch_moddown_f(const Context& c, const ModDownNttJob* jobs, int njobs, int max_out, cudaStream_t s) {
    if (c.np <= 4)
        launch_moddown_k<LOGN, FMA, 4>(c, jobs, njobs, max_out, s);
    else if (c.np <= 8)
        launch_moddown_k<LOGN, FMA, 8>(c, jobs, njobs, max_out, s);
    else
        launch_moddown_k<LOGN, FMA, kMaxPLimbs>(c, jobs, njobs, max_out, s);
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
