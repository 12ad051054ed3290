// CPU emulation of the device kernels (test infrastructure).
//
// Compiles the product's kernel bodies (wg_ntt.cuh, wg_keyswitch.cuh) and host table builder
// (wg_tables.cpp, wg_host.cpp) with the host compiler and runs them CTA by CTA and thread by
// thread, so the index logic, butterflies, HPS base changes and tables can be checked against
// the oracle without a GPU.  Shared-memory rounds are separated exactly where the kernels put
// __syncthreads().  Not part of the product library.
#include <array>
#include <cstring>
#include <type_traits>
#include <utility>
#include <stdexcept>
#include <vector>

#include "wg_keyswitch.cuh"
#include "wg_ksfuse.cuh"
#include "wg_ntt.cuh"
#include "wg_tables.hpp"
#include "wg_tensor.cuh"
#include "wg_walsh.cuh"
#include "wg_ring.hpp"
#include "wg_bundle.hpp"
#include "wg_batching.hpp"
#include <deque>
#include <random>

using namespace wg;

namespace {

struct HostModUp {
    int src_count, dst_count, src_first, pad;
    const uint64_t *qhat_inv, *qhat_inv_s;
    const double* src_inv;
    const uint64_t *qhat, *qhat_s, *corr;
    const int *dst_limb, *dst_mod;
    const ntt::TwPair *scale_fp, *qhat_fp;
};

struct Emu {
    HostTables H;
    int logN;
    std::vector<std::vector<HostModUp>> modup;
    std::vector<ntt::TwPair> tw;  // twiddle pairs of every modulus: [mod][fwd N, inv N]
};

// A modulus's table of one direction as the device makes it (k_twiddles_8, k_twiddles_16), from its split
// words (w at i, its Shoup companion at N + i).
void twiddle_table(int logN, uint64_t q, const uint64_t* w, int eb, ntt::TwPair* out) {
    const size_t N = (size_t)1 << logN;
    for (size_t i = 0; i < N; ++i) out[ntt::twiddle_place(logN, eb, i)] = ntt::twiddle_pair(w[i], w[N + i], q, false);
}

// The rounds of one phase over a CTA: v[t] are thread t's elements, exchanged through the padded tile
// where the kernels do (ntt_round, wg_ntt.cu).
template <class Arith, int E>
using Lanes = std::vector<std::array<typename Arith::V, E>>;

template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL, int RD, class Arith>
void one_round(uint64_t* sm, Lanes<Arith, 1 << EB>& v, int tile, const Arith& ar, const ntt::TwPair* tw) {
    using R = ntt::Round<LOGN, FWD, COLS, EB, STAGED, RD, TL>;
    using P = typename R::P;
    if constexpr (RD > 0) {
        for (int t = 0; t < P::THREADS; ++t)
            ntt::Round<LOGN, FWD, COLS, EB, STAGED, RD - 1, TL>::template scatter<Arith>(sm, P::sub_of(t), P::o_of(t),
                                                                                       v[t].data());
        for (int t = 0; t < P::THREADS; ++t) R::template gather<Arith>(sm, P::sub_of(t), P::o_of(t), v[t].data());
    }
    for (int t = 0; t < P::THREADS; ++t) R::stages(v[t].data(), P::sub_of(t), P::o_of(t), tile, ar, tw);
}
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL, class Arith, int... RD>
void rounds(std::integer_sequence<int, RD...>, uint64_t* sm, Lanes<Arith, 1 << EB>& v, int tile, const Arith& ar,
            const ntt::TwPair* tw) {
    (one_round<LOGN, FWD, COLS, EB, STAGED, TL, RD>(sm, v, tile, ar, tw), ...);
}

// A limb's tile through one phase: `in` maps a word of the limb to the rounds' bits, `out` back.
template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED, int TL, class Arith, class In, class Out>
void tile_phase(uint64_t* x, int tile, const Arith& ar, const ntt::TwPair* tw, In in, Out out) {
    using P = ntt::Phase<LOGN, FWD, COLS, EB, STAGED, TL>;
    using Begin = ntt::Round<LOGN, FWD, COLS, EB, STAGED, 0, TL>;
    using End = ntt::Round<LOGN, FWD, COLS, EB, STAGED, P::ROUNDS - 1, TL>;
    std::vector<uint64_t> sm(P::TILE + P::TILE / 16);
    Lanes<Arith, 1 << EB> v(P::THREADS);
    for (int t = 0; t < P::THREADS; ++t) {
        const uint64_t* p = x + ntt::tile_offset<LOGN, FWD, COLS, EB, STAGED, TL>(tile, Begin::element(P::sub_of(t), P::o_of(t)));
        for (int j = 0; j < P::E; ++j) v[t][j] = Arith::of_bits(in(p[Begin::limb_step(j)]));
    }
    rounds<LOGN, FWD, COLS, EB, STAGED, TL>(std::make_integer_sequence<int, P::ROUNDS>{}, sm.data(), v, tile, ar, tw);
    for (int t = 0; t < P::THREADS; ++t) {
        uint64_t* p = x + ntt::tile_offset<LOGN, FWD, COLS, EB, STAGED, TL>(tile, End::element(P::sub_of(t), P::o_of(t)));
        for (int j = 0; j < P::E; ++j) p[End::limb_step(j)] = out(Arith::bits(v[t][j]));
    }
}

using ntt::word_store;

// NTT geometry the emulated phases use (the device's kNttGeometries order: 0 = 8 residues per
// thread, staged twiddles; 1 = 8, table; 2 = 16, staged; 3 = 16, table).
int g_geometry = 0;

template <int LOGN, bool FWD, bool COLS, int EB, bool STAGED>
void phase(const Emu& E, uint64_t* x, int mi, bool epilogue) {
    using P = ntt::Phase<LOGN, FWD, COLS, EB, STAGED>;
    const size_t N = P::N;
    std::vector<ntt::TwPair> table(N);
    const uint64_t* w = E.H.tw.data() + ((size_t)mi * 4 + (FWD ? 0 : 2)) * N;
    twiddle_table(E.logN, E.H.mods[mi].q, w, EB, table.data());
    const ntt::TwPair* tw = table.data();
    const Modulus& md = E.H.mods[mi];
    const bool fp64 = md.q < fp::kLimit, lazy = FWD && md.q < ntt::kLazyForwardLimit;
    const bool first = FWD ? COLS : !COLS;
    std::vector<ntt::TwPair> tw_s(P::TW);
    const auto out = [&](uint64_t v) { return word_store(P::LAST, FWD, v, md); };
    const auto same = [](uint64_t v) { return v; };
    for (int tile = 0; tile < (int)(N / P::TILE); ++tile) {
        if (STAGED)
            for (int e = 0; e < P::TW; ++e) tw_s[e] = tw[ntt::twiddle_src<LOGN, FWD, COLS, EB, STAGED>(tile, e)];
        const ntt::TwPair* twr = STAGED ? tw_s.data() : tw;
        if (fp64)
            tile_phase<LOGN, FWD, COLS, EB, STAGED, ntt::kMaxTile>(
                x, tile, ntt::fp_arith(md), twr, [&](uint64_t v) { return ntt::fp_load(first, v, md); },
                [&](uint64_t v) { return epilogue ? v : ntt::fp_store(P::LAST, FWD, v, md); });
        else if (lazy)
            tile_phase<LOGN, FWD, COLS, EB, STAGED, ntt::kMaxTile>(x, tile, ntt::WordArith<true>{md.q}, twr, same, out);
        else
            tile_phase<LOGN, FWD, COLS, EB, STAGED, ntt::kMaxTile>(x, tile, ntt::WordArith<false>{md.q}, twr, same, out);
    }
}

// epilogue: leave an FP64 limb's last words to the caller's epilogue (k_ntt_rows_epi)
template <int LOGN, bool FWD, bool COLS>
void phase_geom(const Emu& E, uint64_t* x, int mi, bool epilogue = false) {
    switch (g_geometry) {
        case 0: phase<LOGN, FWD, COLS, 3, true>(E, x, mi, epilogue); break;
        case 1: phase<LOGN, FWD, COLS, 3, false>(E, x, mi, epilogue); break;
        case 2: phase<LOGN, FWD, COLS, 4, true>(E, x, mi, epilogue); break;
        default: phase<LOGN, FWD, COLS, 4, false>(E, x, mi, epilogue); break;
    }
}

template <int LOGN>
void ntt_limb(const Emu& E, uint64_t* x, int mi, bool fwd) {
    if (fwd) {
        phase_geom<LOGN, true, true>(E, x, mi);
        phase_geom<LOGN, true, false>(E, x, mi);
    } else {
        phase_geom<LOGN, false, false>(E, x, mi);
        phase_geom<LOGN, false, true>(E, x, mi);
    }
}

void ntt_one(const Emu& E, uint64_t* x, int mi, bool fwd) {
    switch (E.logN) {
        case 10: ntt_limb<10>(E, x, mi, fwd); break;
        case 11: ntt_limb<11>(E, x, mi, fwd); break;
        case 12: ntt_limb<12>(E, x, mi, fwd); break;
        case 13: ntt_limb<13>(E, x, mi, fwd); break;
        case 14: ntt_limb<14>(E, x, mi, fwd); break;
        case 15: ntt_limb<15>(E, x, mi, fwd); break;
        case 16: ntt_limb<16>(E, x, mi, fwd); break;
        default: throw std::invalid_argument("emu: unsupported ring degree");
    }
}

// Key switches and rescales run the fused sequences of wg_ksfuse.cu (Context::ntt_fusion), each job's
// outputs over g_fused blocks a column tile (split_of).
int g_fused = 0;

bool is_fp(const Emu& E, int mi) { return E.H.mods[mi].q < fp::kLimit; }

template <class G, bool FWD, class Arith>
void columns(Lanes<Arith, G::E>& v, int tile, const Arith& ar, const ntt::TwPair* tw) {
    std::vector<uint64_t> sm(G::PAD);
    rounds<G::LOG, FWD, true, G::BITS, false, ksf::kTile>(std::make_integer_sequence<int, G::ROUNDS>{}, sm.data(), v, tile, ar, tw);
}

// inverse_slots (wg_ksfuse.cu) of one source limb whose words thread t has at slots[k * THREADS + t].
template <class G, class ScaleFp, class ScaleWords>
void inverse_slots(const Emu& E, uint64_t* slots, int tile, int mi, ScaleFp scale_f, ScaleWords scale_w) {
    const Modulus& m = E.H.mods[mi];
    const ntt::TwPair* tw = E.tw.data() + (size_t)mi * 2 * G::N + G::N;
    auto run = [&](const auto& ar, auto scale) {
        using A = std::decay_t<decltype(ar)>;
        Lanes<A, G::E> v(G::THREADS);
        for (int t = 0; t < G::THREADS; ++t)
            for (int k = 0; k < G::E; ++k) v[t][k] = A::of_bits(slots[k * G::THREADS + t]);
        columns<G, false>(v, tile, ar, tw);
        for (int t = 0; t < G::THREADS; ++t) {
            scale(v[t].data(), t);
            for (int k = 0; k < G::E; ++k) slots[k * G::THREADS + t] = A::bits(v[t][k]);
        }
    };
    if (is_fp(E, mi))
        run(ntt::fp_arith(m), scale_f);
    else
        run(ntt::WordArith<false>{m.q}, scale_w);
}
template <class G>
void load_slots(uint64_t* slots, const uint64_t* limb, int tile) {
    for (int t = 0; t < G::THREADS; ++t) {
        uint64_t w[G::E];
        ksf::load_limb<typename G::template InvRound<0>>(w, limb, tile, t);
        for (int k = 0; k < G::E; ++k) slots[k * G::THREADS + t] = w[k];
    }
}
// forward_limb (wg_ksfuse.cu).
template <class G, class ValueFp, class ValueWords>
void forward_limb(const Emu& E, uint64_t* limb, int tile, int mi, ValueFp value_f, ValueWords value_w) {
    using End = typename G::template FwdRound<G::ROUNDS - 1>;
    const Modulus& m = E.H.mods[mi];
    const ntt::TwPair* tw = E.tw.data() + (size_t)mi * 2 * G::N;
    auto run = [&](const auto& ar, auto value) {
        using A = std::decay_t<decltype(ar)>;
        Lanes<A, G::E> v(G::THREADS);
        for (int t = 0; t < G::THREADS; ++t) value(v[t].data(), t);
        columns<G, true>(v, tile, ar, tw);
        for (int t = 0; t < G::THREADS; ++t) {
            uint64_t w[G::E];
            for (int k = 0; k < G::E; ++k) w[k] = A::bits(v[t][k]);
            ksf::store_limb<End>(w, limb, tile, t);
        }
    };
    if (is_fp(E, mi))
        run(ntt::fp_arith(m), value_f);
    else if (m.q < ntt::kLazyForwardLimit)
        run(ntt::WordArith<true>{m.q}, value_w);
    else
        run(ntt::WordArith<false>{m.q}, value_w);
}

// k_modup_ntt over every column tile of one digit.
template <class G>
void modup_fused_g(const Emu& E, const HostModUp& d, const uint64_t* src, uint64_t* digit) {
    const int n = d.src_count;
    std::vector<uint64_t> slots((size_t)n * G::TILE);
    for (int block = 0; block < G::TILES * g_fused; ++block) {
        const ksf::Share sh = ksf::share_of(block, G::TILES * g_fused, G::TILES);
        const int tile = sh.tile;
        std::vector<double> alpha((size_t)G::THREADS * G::E, 0.0);
        ksf::SourceKinds kinds;
        for (int i = 0; i < n; ++i) {
            const int mi = d.src_first + i;
            const Modulus& m = E.H.mods[mi];
            uint64_t* sl = slots.data() + (size_t)i * G::TILE;
            kinds.set(i, m.q);
            load_slots<G>(sl, src + (size_t)mi * G::N, tile);
            inverse_slots<G>(
                E, sl, tile, mi,
                [&](double* v, int t) { ksf::modup_scale_fp<G>(v, d, i, m.qd, alpha.data() + (size_t)t * G::E); },
                [&](uint64_t* v, int t) {
                    ksf::scale_n_inv<G::E>(v, m);
                    ksf::modup_scale<G>(v, d, i, m.q, alpha.data() + (size_t)t * G::E);
                });
        }
        std::vector<uint32_t> hps((size_t)G::THREADS * G::E);
        for (size_t k = 0; k < hps.size(); ++k) hps[k] = ksf::hps_count(alpha[k], n);
        for (int dst = sh.begin; dst < d.dst_count; dst += sh.step) {
            const int mi = d.dst_mod[dst];
            const Modulus& m = E.H.mods[mi];
            forward_limb<G>(
                E, digit + (size_t)d.dst_limb[dst] * G::N, tile, mi,
                [&](double* v, int t) {
                    ksf::modup_value_fp<G>(v, slots.data(), t, d, dst, m, hps.data() + (size_t)t * G::E, kinds);
                },
                [&](uint64_t* v, int t) {
                    ksf::modup_value<G>(v, slots.data(), t, d, dst, m.q, hps.data() + (size_t)t * G::E, kinds.fp64);
                });
        }
    }
}
template <int LOGN>
void modup_fused(const Emu& E, const HostModUp& d, const uint64_t* src, uint64_t* digit) {
    bool words = false;  // Context::word_moduli
    for (const Modulus& m : E.H.mods) words |= m.q >= fp::kLimit;
    if (words)
        modup_fused_g<ksf::Geom<LOGN, ksf::kModUpBits>>(E, d, src, digit);
    else
        modup_fused_g<ksf::Geom<LOGN, ksf::kModUpFpBits>>(E, d, src, digit);
}

// k_moddown_ntt over every column tile of one accumulator polynomial.
template <int LOGN>
void moddown_fused(const Emu& E, const uint64_t* src_p, uint64_t* out, int L, const uint64_t* inv,
                   const uint64_t* inv_s, const ntt::TwPair* inv_fp) {
    using G = ksf::Geom<LOGN, ksf::kModDownBits>;
    const int K = (int)E.H.np, nq = (int)E.H.nq;
    const Modulus* pmods = E.H.mods.data() + nq;
    std::vector<uint64_t> slots((size_t)K * G::TILE);
    ksf::SourceKinds kinds;
    for (int pi = 0; pi < K; ++pi) kinds.set(pi, pmods[pi].q);
    for (int block = 0; block < G::TILES * g_fused; ++block) {
        const ksf::Share sh = ksf::share_of(block, G::TILES * g_fused, G::TILES);
        const int tile = sh.tile;
        for (int pi = 0; pi < K; ++pi) {
            const Modulus& m = pmods[pi];
            uint64_t* sl = slots.data() + (size_t)pi * G::TILE;
            load_slots<G>(sl, src_p + (size_t)pi * G::N, tile);
            inverse_slots<G>(
                E, sl, tile, nq + pi, [&](double* v, int) { ksf::scale_fp<G::E>(v, m.n_inv_w, m.n_inv_wq, m.qd); },
                [&](uint64_t* v, int) { ksf::scale_n_inv<G::E>(v, m); });
        }
        std::vector<uint32_t> hps((size_t)G::THREADS * G::E);
        for (int t = 0; t < G::THREADS; ++t)
            ksf::moddown_hps<G>(slots.data(), t, pmods, K, hps.data() + (size_t)t * G::E, kinds.fp64);
        for (int qi = sh.begin; qi < L; qi += sh.step) {
            const Modulus& m = E.H.mods[qi];
            const uint64_t *iv = inv + (size_t)qi * K, *ivs = inv_s + (size_t)qi * K;
            forward_limb<G>(
                E, out + (size_t)qi * G::N, tile, qi,
                [&](double* v, int t) {
                    ksf::moddown_value_fp<G>(v, slots.data(), t, K, m, iv, ivs, inv_fp + (size_t)qi * K,
                                                hps.data() + (size_t)t * G::E, kinds);
                },
                [&](uint64_t* v, int t) {
                    ksf::moddown_value<G>(v, slots.data(), t, K, m.q, iv, ivs, hps.data() + (size_t)t * G::E, kinds.fp64);
                });
        }
    }
}

// k_rows_mac for one switch: QP limb i of both accumulators from the digits as the fused ModUp leaves
// them (key limb klimb of key_limbs).
template <int LOGN, class Sums, class Fwd, class Inv>
void rows_mac_limb(const Emu& E, const Modulus& m, int mi, int parts, int own_part, const uint64_t* key_term,
                   const uint64_t* digits, size_t part_stride, const uint64_t* key, size_t key_stride, uint64_t* acc_a,
                   uint64_t* acc_b, bool rows, const Fwd& fwd, const Inv& inv) {
    using P = ntt::Phase<LOGN, true, false, 3, false>;
    using Begin = ntt::Round<LOGN, true, false, 3, false, 0>;
    using End = ntt::Round<LOGN, true, false, 3, false, P::ROUNDS - 1>;
    using InvEnd = ntt::Round<LOGN, false, false, 3, false, P::ROUNDS - 1>;
    constexpr auto all = std::make_integer_sequence<int, P::ROUNDS>{};
    const ntt::TwPair* tw = E.tw.data() + (size_t)mi * 2 * P::N;
    std::vector<uint64_t> sm(P::TILE + P::TILE / 16);
    for (int tile = 0; tile < P::N / P::TILE; ++tile) {
        const size_t at = (size_t)tile * P::TILE;
        std::vector<Sums> sums(P::THREADS);
        for (auto& s : sums) s.clear();
        Lanes<Fwd, 8> v(P::THREADS);
        auto element = [&](auto round, int t) { return at + decltype(round)::element(P::sub_of(t), P::o_of(t)); };
        for (int p = 0; p < parts; ++p) {
            const uint64_t* d = digits + p * part_stride;
            for (int t = 0; t < P::THREADS; ++t)
                for (int k = 0; k < 8; ++k)
                    v[t][k] = p == own_part ? Sums::own(key_term[element(End{}, t) + End::limb_step(k)])
                                            : Sums::digit(d[element(Begin{}, t) + Begin::limb_step(k)]);
            if (p != own_part) {
                rounds<LOGN, true, false, 3, false, ntt::kMaxTile>(all, sm.data(), v, tile, fwd, tw);
                for (auto& x : v) Sums::transformed(x.data(), m);
            }
            for (int t = 0; t < P::THREADS; ++t)
                for (int poly = 0; poly < 2; ++poly) {
                    uint64_t k8[8];
                    for (int k = 0; k < 8; ++k)
                        k8[k] = key[(2 * p + poly) * key_stride + element(End{}, t) + End::limb_step(k)];
                    sums[t].add(poly, v[t].data(), k8, p, m);
                }
        }
        for (int poly = 0; poly < 2; ++poly) {
            uint64_t* out = poly ? acc_b : acc_a;
            if (rows) {
                for (int t = 0; t < P::THREADS; ++t)
                    for (int k = 0; k < 8; ++k) v[t][k] = sums[t].value(poly, k, m);
                rounds<LOGN, false, false, 3, false, ntt::kMaxTile>(all, sm.data(), v, tile, inv, tw + P::N);
                for (int t = 0; t < P::THREADS; ++t)
                    for (int k = 0; k < 8; ++k)
                        out[element(InvEnd{}, t) + InvEnd::limb_step(k)] = Sums::row_word(v[t][k], m);
            } else {
                for (int t = 0; t < P::THREADS; ++t)
                    for (int k = 0; k < 8; ++k) out[element(End{}, t) + End::limb_step(k)] = sums[t].word(poly, k, m);
            }
        }
    }
}
template <int LOGN>
void rows_mac(const Emu& E, size_t L, size_t B, const uint64_t* key, size_t key_level, const uint64_t* key_term,
              const uint64_t* digits, uint64_t* acc) {
    const size_t N = E.H.N, K = E.H.np, T = L + K;
    for (size_t i = 0; i < T; ++i) {
        const bool rows = i >= L;
        const int mi = (int)(rows ? E.H.nq + i - L : i), own = rows ? -1 : (int)(i / E.H.alpha);
        const size_t klimb = rows ? key_level + 1 + (i - L) : i, stride = (key_level + 1 + K) * N;
        const Modulus& m = E.H.mods[mi];
        auto run = [&](auto sums, const auto& fwd, const auto& inv) {
            rows_mac_limb<LOGN, decltype(sums)>(E, m, mi, (int)B, own, key_term + (rows ? 0 : i * N), digits + i * N, T * N,
                                               key + klimb * N, stride, acc + i * N, acc + (T + i) * N, rows, fwd, inv);
        };
        if (is_fp(E, mi))
            run(ntt::MacSumsFp{}, ntt::fp_arith(m), ntt::fp_arith(m));
        else if (m.q < ntt::kLazyForwardLimit)
            run(ntt::MacSumsWords{}, ntt::WordArith<true>{m.q}, ntt::WordArith<false>{m.q});
        else
            run(ntt::MacSumsWords{}, ntt::WordArith<false>{m.q}, ntt::WordArith<false>{m.q});
    }
}

// k_ntt_rows_epi for one job: the forward row phase of a copy of the job's limb (the kernel
// reads it and stores nothing back) with the emulated geometry, then the epilogue per word.
template <int LOGN>
void rows_epi(const Emu& E, const ntt::NttEpiJob& j) {
    const size_t N = (size_t)1 << LOGN;
    std::vector<uint64_t> v(j.data, j.data + N);
    phase_geom<LOGN, true, false>(E, v.data(), j.mod, true);
    const Modulus& m = E.H.mods[j.mod];
    if (is_fp(E, j.mod)) {
        const ntt::FpEpilogue c = ntt::fp_epilogue(j, m);
        for (size_t off = 0; off < N; ++off)
            j.out[off] = ntt::fp_epilogue_value(j, c, j.kind == ntt::kEpiCombine ? j.acc[off] : 0,
                                                j.kind == ntt::kEpiRescale || j.c0 ? j.in[off] : 0, v[off], m);
        return;
    }
    for (size_t off = 0; off < N; ++off) ntt::ntt_epilogue(j, off, v[off], m.q);
}

// k_rescale_ntt over every column tile of one polynomial (dropped limb after the inverse row
// phase); rc: the rescale constants of level lv (one_s, inv_p, inv_p_s, half).
template <int LOGN>
void rescale_fused(const Emu& E, const uint64_t* drop, uint64_t* rem, int lv, const uint64_t* rc) {
    using G = ksf::Geom<LOGN, ksf::kRescaleBits>;
    std::vector<uint64_t> slots(G::TILE);
    const Modulus& mp = E.H.mods[lv];
    for (int block = 0; block < G::TILES * g_fused; ++block) {
        const ksf::Share sh = ksf::share_of(block, G::TILES * g_fused, G::TILES);
        const int tile = sh.tile;
        load_slots<G>(slots.data(), drop, tile);
        inverse_slots<G>(
            E, slots.data(), tile, lv, [&](double* v, int) { ksf::scale_fp<G::E>(v, mp.n_inv_w, mp.n_inv_wq, mp.qd); },
            [&](uint64_t* v, int) { ksf::scale_n_inv<G::E>(v, mp); });
        for (int qi = sh.begin; qi < lv; qi += sh.step) {
            const Modulus& m = E.H.mods[qi];
            forward_limb<G>(
                E, rem + (size_t)qi * G::N, tile, qi,
                [&](double* v, int t) {
                    ksf::rescale_value_fp<G>(v, slots.data(), t, mp.q, m, rc[qi], rc[3 * lv + qi], is_fp(E, lv));
                },
                [&](uint64_t* v, int t) {
                    ksf::rescale_value<G>(v, slots.data(), t, mp.q, m.q, rc[qi], rc[3 * lv + qi], is_fp(E, lv));
                });
        }
    }
}

// One phase of one limb with the emulated geometry (cols: the high-bit phase).
template <int LOGN>
void phase_one(const Emu& E, uint64_t* x, int mi, bool fwd, bool cols) {
    if (fwd) {
        if (cols) phase_geom<LOGN, true, true>(E, x, mi);
        else phase_geom<LOGN, true, false>(E, x, mi);
    } else {
        if (cols) phase_geom<LOGN, false, true>(E, x, mi);
        else phase_geom<LOGN, false, false>(E, x, mi);
    }
}

// k_ntt_whole of one limb: every CTA of the cluster runs the first phase on its tile, hands the
// results over (HandOver), then runs the second.
template <int LOGN, bool FWD, class Arith>
void whole_limb(const Emu& E, uint64_t* x, int mi, const Arith& ar) {
    using W = ntt::Whole<LOGN>;
    using P1 = typename W::template Ph<FWD, FWD>;
    using P2 = typename W::template Ph<FWD, !FWD>;
    using Begin1 = ntt::Round<LOGN, FWD, FWD, 3, false, 0, W::TL>;
    using End1 = ntt::Round<LOGN, FWD, FWD, 3, false, P1::ROUNDS - 1, W::TL>;
    using Begin2 = ntt::Round<LOGN, FWD, !FWD, 3, false, 0, W::TL>;
    using End2 = ntt::Round<LOGN, FWD, !FWD, 3, false, P2::ROUNDS - 1, W::TL>;
    const Modulus& m = E.H.mods[mi];
    const bool fp64 = is_fp(E, mi);
    const ntt::TwPair* tw = E.tw.data() + (size_t)mi * 2 * W::N + (FWD ? 0 : W::N);
    std::vector<uint64_t> first(W::PAD), second((size_t)W::CTAS * W::PAD, ~uint64_t{0});
    for (int tile = 0; tile < W::CTAS; ++tile) {
        Lanes<Arith, 8> v(P1::THREADS);
        for (int t = 0; t < P1::THREADS; ++t) {
            const uint64_t* p = x + ntt::tile_offset<LOGN, FWD, FWD, 3, false, W::TL>(
                                        tile, Begin1::element(P1::sub_of(t), P1::o_of(t)));
            for (int j = 0; j < 8; ++j) {
                const uint64_t w = p[Begin1::limb_step(j)];
                v[t][j] = Arith::of_bits(fp64 ? ntt::fp_load(true, w, m) : w);
            }
        }
        rounds<LOGN, FWD, FWD, 3, false, W::TL>(std::make_integer_sequence<int, P1::ROUNDS>{}, first.data(), v, tile, ar, tw);
        for (int t = 0; t < P1::THREADS; ++t)
            for (int j = 0; j < 8; ++j) {
                const ntt::HandOver h = ntt::hand_over<LOGN, FWD>(
                    tile, End1::element(P1::sub_of(t), P1::o_of(t)) + End1::tile_step(j));
                const uint64_t w = Arith::bits(v[t][j]);
                second[(size_t)h.cta * W::PAD + ntt::pad16(h.at)] = fp64 ? ntt::fp_store(false, FWD, w, m) : w;
            }
    }
    for (int tile = 0; tile < W::CTAS; ++tile) {
        Lanes<Arith, 8> v(P2::THREADS);
        for (int t = 0; t < P2::THREADS; ++t)
            Begin2::template gather<Arith>(second.data() + (size_t)tile * W::PAD, P2::sub_of(t), P2::o_of(t), v[t].data());
        rounds<LOGN, FWD, !FWD, 3, false, W::TL>(std::make_integer_sequence<int, P2::ROUNDS>{}, first.data(), v, tile, ar, tw);
        for (int t = 0; t < P2::THREADS; ++t) {
            uint64_t* p = x + ntt::tile_offset<LOGN, FWD, !FWD, 3, false, W::TL>(
                                  tile, End2::element(P2::sub_of(t), P2::o_of(t)));
            for (int j = 0; j < 8; ++j) {
                const uint64_t w = Arith::bits(v[t][j]);
                p[End2::limb_step(j)] = fp64 ? ntt::fp_store(true, FWD, w, m) : word_store(true, FWD, w, m);
            }
        }
    }
}
template <int LOGN>
void whole_ntt(const Emu& E, uint64_t* x, int mi, bool fwd) {
    const Modulus& m = E.H.mods[mi];
    if (is_fp(E, mi))
        fwd ? whole_limb<LOGN, true>(E, x, mi, ntt::fp_arith(m)) : whole_limb<LOGN, false>(E, x, mi, ntt::fp_arith(m));
    else if (fwd && m.q < ntt::kLazyForwardLimit)
        whole_limb<LOGN, true>(E, x, mi, ntt::WordArith<true>{m.q});
    else
        fwd ? whole_limb<LOGN, true>(E, x, mi, ntt::WordArith<false>{m.q})
            : whole_limb<LOGN, false>(E, x, mi, ntt::WordArith<false>{m.q});
}

#define EMU_LOGN_SWITCH(logN, CALL)                                        \
    do switch (logN) {                                                     \
        case 10: { constexpr int LG = 10; CALL; } break;                   \
        case 11: { constexpr int LG = 11; CALL; } break;                   \
        case 12: { constexpr int LG = 12; CALL; } break;                   \
        case 13: { constexpr int LG = 13; CALL; } break;                   \
        case 14: { constexpr int LG = 14; CALL; } break;                   \
        case 15: { constexpr int LG = 15; CALL; } break;                   \
        case 16: { constexpr int LG = 16; CALL; } break;                   \
        default: throw std::invalid_argument("emu: unsupported ring degree"); \
    } while (0)

}  // namespace

extern "C" {

void* emu_create(uint64_t N, const uint64_t* q, size_t nq, const uint64_t* p, size_t np, size_t dnum) {
    Emu* E = new Emu;
    E->H = build_tables(N, q, nq, p, np, dnum);
    E->logN = __builtin_ctzll(N);
    const uint64_t* T = E->H.words.data();
    E->modup.resize(nq);
    for (size_t l = 0; l < nq; ++l)
        for (const auto& o : E->H.modup[l]) {
            HostModUp d;
            d.src_count = o.src_count;
            d.dst_count = o.dst_count;
            d.src_first = o.src_first;
            d.pad = 0;
            d.qhat_inv = T + o.qhat_inv;
            d.qhat_inv_s = T + o.qhat_inv_s;
            d.src_inv = reinterpret_cast<const double*>(T + o.src_inv);
            d.qhat = T + o.qhat;
            d.qhat_s = T + o.qhat_s;
            d.corr = T + o.corr;
            d.dst_limb = reinterpret_cast<const int*>(T + o.dst_limb);
            d.dst_mod = reinterpret_cast<const int*>(T + o.dst_mod);
            d.scale_fp = reinterpret_cast<const ntt::TwPair*>(T + o.scale_fp);
            d.qhat_fp = reinterpret_cast<const ntt::TwPair*>(T + o.qhat_fp);
            E->modup[l].push_back(d);
        }
    E->tw.resize((nq + np) * 2 * N);
    for (size_t m = 0; m < nq + np; ++m)
        for (size_t dir = 0; dir < 2; ++dir) {
            const uint64_t* w = E->H.tw.data() + (m * 4 + 2 * dir) * N;
            twiddle_table(E->logN, E->H.mods[m].q, w, 3, E->tw.data() + (m * 2 + dir) * N);
        }
    return E;
}

void emu_destroy(void* h) { delete static_cast<Emu*>(h); }

void emu_set_ntt_geometry(int geometry) { g_geometry = geometry; }
void emu_set_keyswitch_fusion(int fused) { g_fused = fused; }

// limbs consecutive limbs using modulus index first.. (basis 0 = Q, 1 = P)
void emu_ntt(void* h, uint64_t* poly, size_t limbs, size_t first, int basis, int inverse) {
    const Emu& E = *static_cast<Emu*>(h);
    for (size_t l = 0; l < limbs; ++l)
        ntt_one(E, poly + l * E.H.N, (int)((basis ? E.H.nq : 0) + first + l), !inverse);
}

// The same through the one-launch transforms.
void emu_ntt_whole(void* h, uint64_t* poly, size_t limbs, size_t first, int basis, int inverse) {
    const Emu& E = *static_cast<Emu*>(h);
    for (size_t l = 0; l < limbs; ++l) {
        uint64_t* x = poly + l * E.H.N;
        const int mi = (int)((basis ? E.H.nq : 0) + first + l);
        switch (E.logN) {
            case 10: whole_ntt<10>(E, x, mi, !inverse); break;
            case 11: whole_ntt<11>(E, x, mi, !inverse); break;
            case 12: whole_ntt<12>(E, x, mi, !inverse); break;
            case 13: whole_ntt<13>(E, x, mi, !inverse); break;
            case 14: whole_ntt<14>(E, x, mi, !inverse); break;
            default: throw std::invalid_argument("emu: ring too large for the one-launch transform");
        }
    }
}

// The device keyswitch() sequence, stage by stage, with the same buffers.
void emu_keyswitch(void* h, size_t level, const uint64_t* key_term, const uint64_t* key, size_t key_level,
                   uint64_t* b, uint64_t* a, int b_add, int a_add, uint64_t galois) {
    const Emu& E = *static_cast<Emu*>(h);
    const size_t N = E.H.N, L = level + 1, K = E.H.np, T = L + K, nq = E.H.nq;
    const size_t alpha = E.H.alpha;
    const size_t B = parts_at(level, nq, alpha, E.H.dnum);
    std::vector<uint64_t> ws(N * (L + B * T + 2 * T + 2 * L));
    uint64_t* coeff = ws.data();
    uint64_t* digits = coeff + L * N;
    uint64_t* acc = digits + B * T * N;
    uint64_t* contrib = acc + 2 * T * N;
    const Modulus* mods = E.H.mods.data();
    std::memcpy(coeff, key_term, L * N * 8);
    if (g_fused) {
        // inverse row phase, fused [inverse columns, ModUp, forward columns]
        for (size_t l = 0; l < L; ++l) EMU_LOGN_SWITCH(E.logN, phase_one<LG>(E, coeff + l * N, (int)l, false, false));
        for (size_t j = 0; j < B; ++j)
            EMU_LOGN_SWITCH(E.logN, modup_fused<LG>(E, E.modup[level][j], coeff, digits + j * T * N));
    } else {
        for (size_t l = 0; l < L; ++l) ntt_one(E, coeff + l * N, (int)l, false);
        for (size_t j = 0; j < B; ++j)
            for (size_t c = 0; c < N; ++c) modup_coeff(E.modup[level][j], mods, coeff, digits + j * T * N, N, c);
    }
    if (g_fused) {
        // fused [forward row phase, key product, inverse row phase of the P limbs]
        EMU_LOGN_SWITCH(E.logN, rows_mac<LG>(E, L, B, key, key_level, key_term, digits, acc));
    } else {
        for (size_t j = 0; j < B; ++j) {
            const size_t s0 = j * alpha, s1 = std::min(s0 + alpha, L);
            for (size_t l = 0; l < T; ++l)
                if (l < s0 || l >= s1) ntt_one(E, digits + j * T * N + l * N, (int)(l < L ? l : nq + (l - L)), true);
        }
        for (size_t i = 0; i < T; ++i)
            for (size_t c = 0; c < N; ++c)
                mac_coeff(mods, (int)nq, (int)L, (int)K, (int)B, (int)alpha, key, (int)key_level, key_term, digits, T * N,
                          acc, N, (int)i, c);
    }
    const uint64_t* W = E.H.words.data();
    if (g_fused) {
        for (int poly = 0; poly < 2; ++poly)
            EMU_LOGN_SWITCH(E.logN, moddown_fused<LG>(E, acc + (poly * T + L) * N, contrib + poly * L * N, (int)L,
                                                      W + E.H.fold_inv[level], W + E.H.fold_inv_s[level],
                                                      reinterpret_cast<const ntt::TwPair*>(W + E.H.fold_fp[level])));
        // forward row phase of the contributions with the combine as its epilogue (outputs over
        // the accumulators' Q limbs when an automorphism follows)
        const bool gal = galois != 0;
        for (size_t qi = 0; qi < L; ++qi) {
            const ntt::NttEpiJob ja{contrib + qi * N, acc + qi * N, a + qi * N, (gal ? acc : a) + qi * N,
                                    (uint64_t)a_add, 0, (int)qi, ntt::kEpiCombine};
            const ntt::NttEpiJob jb{contrib + (L + qi) * N, acc + (T + qi) * N, b + qi * N,
                                    (gal ? acc + T * N : b) + qi * N, (uint64_t)b_add, 0, (int)qi, ntt::kEpiCombine};
            EMU_LOGN_SWITCH(E.logN, rows_epi<LG>(E, ja));
            EMU_LOGN_SWITCH(E.logN, rows_epi<LG>(E, jb));
        }
        if (gal)
            for (size_t qi = 0; qi < L; ++qi)
                for (uint32_t i = 0; i < N; ++i) {
                    const uint32_t s = automorphism_src(i, galois, E.logN);
                    b[qi * N + i] = acc[(T + qi) * N + s];
                    a[qi * N + i] = acc[qi * N + s];
                }
        return;
    } else {
        for (int poly = 0; poly < 2; ++poly)
            for (size_t pi = 0; pi < K; ++pi) ntt_one(E, acc + (poly * T + L + pi) * N, (int)(nq + pi), false);
        for (int poly = 0; poly < 2; ++poly)
            for (size_t c = 0; c < N; ++c)
                moddown_all_limbs(mods, (int)nq, (int)L, (int)K, acc + (poly * T + L) * N, N, c,
                                  W + E.H.fold_inv[level], W + E.H.fold_inv_s[level], contrib + poly * L * N);
        for (int poly = 0; poly < 2; ++poly)
            for (size_t qi = 0; qi < L; ++qi) ntt_one(E, contrib + (poly * L + qi) * N, (int)qi, true);
    }
    if (galois == 0) {
        for (size_t qi = 0; qi < L; ++qi)
            for (size_t c = 0; c < N; ++c)
                combine_coeff(mods[qi].q, (int)L, (int)K, acc, contrib, b, a, b, a, b_add, a_add, N, (int)qi, c);
    } else {
        uint64_t* tb = acc + T * N;
        uint64_t* ta = acc;
        for (size_t qi = 0; qi < L; ++qi)
            for (size_t c = 0; c < N; ++c)
                combine_coeff(mods[qi].q, (int)L, (int)K, acc, contrib, b, a, tb, ta, b_add, a_add, N, (int)qi, c);
        for (size_t qi = 0; qi < L; ++qi)
            for (uint32_t i = 0; i < N; ++i) {
                const uint32_t s = automorphism_src(i, galois, E.logN);
                b[qi * N + i] = tb[qi * N + s];
                a[qi * N + i] = ta[qi * N + s];
            }
    }
}

// The device rescale sequence (wg_batch_kernels.cuh RescaleJobs) on one polynomial at level lv:
// x holds lv + 1 limbs; afterwards its first lv limbs are the rescaled polynomial.
void emu_rescale(void* h, size_t lv, uint64_t* x) {
    const Emu& E = *static_cast<Emu*>(h);
    const size_t N = E.H.N;
    const uint64_t* rc = E.H.words.data() + E.H.rescale[lv];
    std::vector<uint64_t> rem(lv * N);
    uint64_t* dl = x + lv * N;
    if (g_fused) {
        EMU_LOGN_SWITCH(E.logN, phase_one<LG>(E, dl, (int)lv, false, false));
        EMU_LOGN_SWITCH(E.logN, rescale_fused<LG>(E, dl, rem.data(), (int)lv, rc));
        for (size_t q = 0; q < lv; ++q) {
            const ntt::NttEpiJob j{rem.data() + q * N, nullptr, x + q * N, x + q * N, rc[lv + q], rc[2 * lv + q],
                                   (int)q, ntt::kEpiRescale};
            EMU_LOGN_SWITCH(E.logN, rows_epi<LG>(E, j));
        }
        return;
    }
    ntt_one(E, dl, (int)lv, false);
    const Modulus& mp = E.H.mods[lv];
    for (size_t q = 0; q < lv; ++q) {
        const Modulus& mq = E.H.mods[q];
        uint64_t* r = rem.data() + q * N;
        for (size_t k = 0; k < N; ++k) {  // kb_rescale_prep
            uint64_t shift = dl[k] + (mp.q >> 1);
            if (shift >= mp.q) shift -= mp.q;
            r[k] = sub_mod(reduce_shoup(shift, mq.q, rc[q]), rc[3 * lv + q], mq.q);
        }
        ntt_one(E, r, (int)q, true);
        for (size_t k = 0; k < N; ++k) {  // kb_rescale_finish
            uint64_t v = x[q * N + k];
            if (v >= mq.q) v -= mq.q;
            x[q * N + k] = mul_shoup(sub_mod(v, r[k], mq.q), rc[lv + q], rc[2 * lv + q], mq.q);
        }
    }
}

static Modulus emu_modulus(uint64_t q) {
    Modulus m{};
    const unsigned __int128 mu = ~(unsigned __int128)0 / q;
    m.q = q;
    m.mu_lo = (uint64_t)mu;
    m.mu_hi = (uint64_t)(mu >> 64);
    m.inv_q = 1.0 / (double)q;
    m.qd = (double)q;
    return m;
}

// mont_mul (the Montgomery product of the key inner products) on n pairs: out[i] = x[i] y[i] 2^-64
// mod q for odd q, qninv = -q^-1 mod 2^64 by Newton iteration.
void emu_mont_mul(uint64_t q, const uint64_t* x, const uint64_t* y, size_t n, uint64_t* out) {
    uint64_t inv = q;  // q q = 1 (mod 8): three correct bits, doubled by each step
    for (int k = 0; k < 5; ++k) inv *= 2 - q * inv;
    for (size_t i = 0; i < n; ++i) out[i] = mont_mul(x[i], y[i], q, 0 - inv);
}

// WideSum and the exact FP64 sum (fp::Dot, q < fp::kNoReduce) of n products x[i] y[i], times 2^-64
// modulo q (qninv as in emu_mont_mul): out[0] and out[1].
void emu_mont_sums(uint64_t q, const uint64_t* x, const uint64_t* y, size_t n, uint64_t* out) {
    Modulus m = emu_modulus(q);
    uint64_t inv = q;
    for (int k = 0; k < 5; ++k) inv *= 2 - q * inv;
    m.qninv = 0 - inv;
    uint64_t r_inv = mont_mul(1, 1, q, m.qninv);  // 2^-64 mod q
    fp::factor(r_inv, q, m.r_inv_w, m.r_inv_wq);
    WideSum w;
    w.clear();
    fp::Dot d;
    d.clear();
    for (size_t i = 0; i < n; ++i) {
        w.add(x[i], y[i], m);
        if (q < fp::kNoReduce) {
            d.add(fp::from_word(x[i]), fp::from_word(y[i]));
            if ((i + 1) % fp::kDotTerms == 0) d.carry(m.qd, m.inv_q);
        }
    }
    out[0] = w.mont_value(m);
    out[1] = q < fp::kNoReduce ? fp::mont_sum_word(d.value(m.qd, m.inv_q), m) : out[0];
}

// fp::mulmod on n pairs (a[i] any integer-valued double, w[i] a residue): the representative and,
// in word[i], the canonical word of it.
void emu_fp_mulmod(uint64_t q, const double* a, const uint64_t* w, size_t n, double* out, uint64_t* word) {
    for (size_t i = 0; i < n; ++i) {
        double fw, fwq;
        fp::factor(w[i], q, fw, fwq);
        out[i] = fp::mulmod(a[i], fw, fwq, (double)q);
        word[i] = fp::canonical(out[i], (double)q, 1.0 / (double)q);
    }
}

// The tensor of n coefficients as kb_tensor forms it (out: c2, b1, a1 of each) and in words (ref);
// returns how many went through FP64.
size_t emu_tensor(uint64_t q, const uint64_t* xa, const uint64_t* xb, const uint64_t* ya, const uint64_t* yb, size_t n,
                  uint64_t* out, uint64_t* ref) {
    const Modulus m = emu_modulus(q);
    size_t taken = 0;
    for (size_t i = 0; i < n; ++i, out += 3, ref += 3) {
        out[2] = ref[2] = xa[i];
        out[1] = ref[1] = xb[i];
        const bool fp64 = q < fp::kNoReduce && tensor_fp(out[2], out[1], ya[i], yb[i], out[0], m, tensor_shift(m));
        if (!fp64) tensor_words(out[2], out[1], ya[i], yb[i], out[0], m);
        tensor_words(ref[2], ref[1], ya[i], yb[i], ref[0], m);
        taken += fp64;
    }
    return taken;
}

void emu_fp_reduce(uint64_t q, const double* x, size_t n, double* out) {
    for (size_t i = 0; i < n; ++i) out[i] = fp::reduce(x[i], (double)q, 1.0 / (double)q);
}

// reduce128 on n values (hi[i], lo[i]) modulo q
void emu_reduce128(uint64_t q, const uint64_t* hi, const uint64_t* lo, size_t n, uint64_t* out) {
    const Modulus m = emu_modulus(q);
    for (size_t i = 0; i < n; ++i) out[i] = reduce128(hi[i], lo[i], m);
}

// The fused Walsh products at n residue positions of one limb (limb index 0, modulus q).
// low_b, low_a, high_b, high_a: [n][16] (mask 0 ignored); coefs: [2][16][16] int8; c0: [2][16];
// out: [n][5] = acc b, acc a, raw b, raw a, raw c2.
void emu_walsh_products(uint64_t q, size_t n, const uint64_t* low_b, const uint64_t* low_a, const uint64_t* high_b,
                        const uint64_t* high_a, const uint64_t* pt_i, const int8_t* coefs, const uint64_t* c0,
                        uint64_t* out) {
    const Modulus m = emu_modulus(q);
    WalshCoefs cf{};
    // [2][16][16] signed coefficients, stored biased as in the device table
    uint8_t biased[2 * 16 * 16];
    for (int i = 0; i < 2 * 16 * 16; ++i) biased[i] = (uint8_t)(coefs[i] + kWalshBias);
    std::memcpy(cf.cw, biased, sizeof(cf.cw));
    for (int r = 0; r < 2; ++r)
        for (int hm = 0; hm < kWalshMasks; ++hm) {
            cf.c0[r][hm][0] = c0[r * kWalshMasks + hm];
            for (int lm = 1; lm < kWalshMasks; ++lm)
                cf.cd[hm][lm][r] = coefs[(r * kWalshMasks + hm) * kWalshMasks + lm];
        }
    for (size_t i = 0; i < n; ++i) {
        if (q < fp::kNoReduce) {
            WalshFp f;
            walsh_load_fp(low_b + i * 16, low_a + i * 16, pt_i[i], m, f);
            uint64_t* o = out + i * 5;
            double xb, xa;
            walsh_pair_fp(f, cf, 0, 0, m, xb, xa);
            o[0] = walsh_word(xb, m);
            o[1] = walsh_word(xa, m);
            WalshRaw raw;
            raw.b.clear();
            raw.a.clear();
            raw.c.clear();
            for (int hm = 1; hm < kWalshMasks; ++hm)
                walsh_product_fp(f, cf, hm, 0, m, high_b[i * 16 + hm], high_a[i * 16 + hm], raw);
            o[2] = walsh_word(raw.b.value(m.qd, m.inv_q), m);
            o[3] = walsh_word(raw.a.value(m.qd, m.inv_q), m);
            o[4] = walsh_word(raw.c.value(m.qd, m.inv_q), m);
            continue;
        }
        WalshLow w;
        walsh_load_low(low_b + i * 16, low_a + i * 16, w);
        uint64_t* o = out + i * 5;
        walsh_constant_pair(w, cf, 0, pt_i[i], m, o, o + 1);
        for (int hm = 1; hm < kWalshMasks; ++hm)
            walsh_product(w, cf, hm, 0, pt_i[i], m, high_b[i * 16 + hm], high_a[i * 16 + hm], o + 2, o + 3, o + 4);
    }
}

int emu_whole_launch(int logN, size_t transforms, int sms, int words) { return ntt::whole_launch(logN, transforms, sms, words != 0); }
int emu_launch_geometry(int tuned, int cols, size_t residues, int sms, int words) {
    return ntt::launch_geometry(tuned, cols != 0, residues, sms, words != 0);
}

// The staging ring's placement (wg_ring.hpp) over `steps` seeded uploads of mixed sizes (1 in 100
// a large one), with no upload ever completing on its own (the host arbitrarily far ahead of the
// device): returns how many regions overlapped an upload the placement did not wait for.
size_t emu_ring_violations(uint64_t seed, size_t steps) {
    struct F {
        size_t begin, end;
    };
    std::mt19937_64 g(seed);
    std::deque<F> flights;
    size_t ring = 0, head = 0, bad = 0;
    for (size_t i = 0; i < steps; ++i) {
        const size_t bytes = (g() % 100 == 0) ? (size_t{100} << 20) : (size_t)(1024 + g() % (128 * 1024));
        const size_t need = (bytes + 255) & ~size_t{255};
        if (need > ring) {  // growth: everything in flight completes first
            flights.clear();
            ring = std::max<size_t>(2 * need, size_t{64} << 20);
            head = 0;
        }
        size_t wait = 0;
        const size_t begin = wg::ring_place(head, ring, need, flights, &wait);
        for (size_t k = 0; k < wait; ++k) flights.pop_front();
        for (const F& f : flights)
            if (f.begin < begin + need && begin < f.end) ++bad;
        flights.push_back({begin, begin + need});
        head = begin + need;
    }
    return bad;
}

// The bundle file format (wg_bundle.hpp): a seeded random bundle survives encode + decode
// unchanged (returns 0), and the reader rejects every damaged variant tried: each single flipped
// byte at `trials` seeded positions, every truncation length tried, a wrong magic and a wrong
// version (returns how many damaged variants it accepted).
int emu_bundle_roundtrip(uint64_t seed) {
    std::mt19937_64 g(seed);
    Bundle b;
    b.N = 1u << 10;
    b.dnum = 3;
    for (int i = 0; i < 5; ++i) b.q.push_back(g());
    for (int i = 0; i < 2; ++i) b.p.push_back(g());
    for (int k = 0; k < 3; ++k) {
        BundleKey key;
        key.kind = (int64_t)(g() % 5);
        key.rotation = (int64_t)(g() % 1000) - 500;
        key.parts = 1 + g() % 3;
        key.key_level = g() % 5;
        key.data.resize(1 + g() % 5000);
        for (auto& w : key.data) w = g();
        b.keys.push_back(key);
    }
    for (int k = 0; k < 2; ++k) {
        BundleStage st;
        st.level = g() % 5;
        st.baby = 1 + g() % 16;
        st.slots = 512;
        st.rescale = g() & 1;
        st.indices.resize(1 + g() % 40);
        for (auto& w : st.indices) w = g() % 512;
        st.diagonals.resize(st.indices.size() * 7);
        for (auto& w : st.diagonals) w = g();
        b.stages.push_back(st);
    }
    const auto bytes = bundle_encode(b);
    const Bundle r = bundle_decode(bytes.data(), bytes.size());
    bool same = r.N == b.N && r.dnum == b.dnum && r.q == b.q && r.p == b.p && r.keys.size() == b.keys.size() &&
                r.stages.size() == b.stages.size();
    for (size_t k = 0; same && k < b.keys.size(); ++k)
        same = r.keys[k].kind == b.keys[k].kind && r.keys[k].rotation == b.keys[k].rotation &&
               r.keys[k].parts == b.keys[k].parts && r.keys[k].key_level == b.keys[k].key_level &&
               r.keys[k].data == b.keys[k].data;
    for (size_t k = 0; same && k < b.stages.size(); ++k)
        same = r.stages[k].level == b.stages[k].level && r.stages[k].baby == b.stages[k].baby &&
               r.stages[k].slots == b.stages[k].slots && r.stages[k].rescale == b.stages[k].rescale &&
               r.stages[k].indices == b.stages[k].indices && r.stages[k].diagonals == b.stages[k].diagonals;
    return same ? 0 : 1;
}

size_t emu_bundle_damage_accepted(uint64_t seed, size_t trials) {
    std::mt19937_64 g(seed);
    Bundle b;
    b.N = 64;
    b.dnum = 2;
    b.q = {g(), g()};
    b.p = {g()};
    BundleKey key;
    key.data.resize(100);
    for (auto& w : key.data) w = g();
    b.keys.push_back(key);
    BundleStage st;
    st.indices = {1, 2};
    st.diagonals.resize(10);
    b.stages.push_back(st);
    const auto good = bundle_encode(b);
    size_t accepted = 0;
    auto accepts = [&](const std::vector<uint8_t>& v) {
        try {
            bundle_decode(v.data(), v.size());
            return true;
        } catch (const std::invalid_argument&) {
            return false;
        }
    };
    for (size_t t = 0; t < trials; ++t) {
        auto v = good;
        v[g() % v.size()] ^= (uint8_t)(1u << (g() % 8));
        accepted += accepts(v);
    }
    for (size_t len = 0; len < good.size(); len += 1 + good.size() / 97)
        accepted += accepts(std::vector<uint8_t>(good.begin(), good.begin() + len));
    auto magic = good;
    magic[0] = 'X';
    accepted += accepts(magic);
    auto version = good;
    version[4] = 2;
    accepted += accepts(version);
    return accepted;
}

// The service's request packing (wg_batching.hpp) on `trials` seeded queues of 0..12 requests of
// 1..max_blocks blocks: returns how many queues broke a property of first fit — positions
// ascending, the oldest request taken, the taken blocks within the slots, every skipped request
// too large for the slots left at its turn — or of batch_full (some request skipped, or the
// slots used up exactly).
size_t emu_first_fit_violations(uint64_t seed, size_t trials) {
    std::mt19937_64 g(seed);
    size_t bad = 0;
    for (size_t t = 0; t < trials; ++t) {
        const size_t max_blocks = 1 + g() % 64;
        std::deque<size_t> q(g() % 13);
        for (auto& n : q) n = 1 + g() % max_blocks;
        const auto id = [](size_t n) { return n; };
        const std::vector<size_t> take = wg::first_fit(q, max_blocks, id);
        bool ok = q.empty() ? take.empty() : (!take.empty() && take[0] == 0);
        size_t used = 0, ti = 0;
        bool skipped = false;
        for (size_t k = 0; k < q.size(); ++k) {
            if (ti < take.size() && take[ti] == k) {
                used += q[k];
                ++ti;
            } else {
                skipped = true;
                ok = ok && used + q[k] > max_blocks;
            }
        }
        ok = ok && ti == take.size() && used <= max_blocks;
        for (size_t k = 1; k < take.size(); ++k) ok = ok && take[k] > take[k - 1];
        ok = ok && wg::batch_full(q, max_blocks, id) == (skipped || used == max_blocks);
        bad += ok ? 0 : 1;
    }
    return bad;
}

}  // extern "C"
