"""The FP64 arithmetic of moduli below 2^50 (csrc/wg_fp.cuh): the product, the transforms at the
edges of their ranges, and key switches whose digits mix FP64 and word moduli.

The CPU tests run the kernels' bodies through the emulation; the GPU tests run the kernels.  All
of it is exact: every comparison is word for word.
"""
import ctypes as C

import numpy as np
import pytest

from test_emulation import emu, test_walsh_products_exact as _walsh_exact, u64p  # noqa: F401

f64p = np.ctypeslib.ndpointer(dtype=np.float64, flags="C_CONTIGUOUS")


def _prime(below, N, step=-1):
    """The nearest prime = 1 (mod 2N) below (or, step = 1, above) `below`."""
    q = below // (2 * N) * (2 * N) + 1
    if step < 0 and q >= below:
        q -= 2 * N
    if step > 0 and q <= below:
        q += 2 * N
    while not all(pow(b, q - 1, q) == 1 for b in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37)):
        q += step * 2 * N
    return q


def _edges(N):
    """Moduli on both sides of the path's limit (2^50) and of its reduction limit (2^42), and a small one."""
    return [_prime(1 << 50, N), _prime(1 << 50, N, 1), _prime(1 << 42, N), _prime(1 << 42, N, 1), _prime(1 << 27, N)]


@pytest.mark.parametrize("q", [_prime(1 << 50, 1 << 15), _prime(1 << 42, 1 << 15, 1), 274876334081, 12289])
def test_product_is_exact_and_bounded(emu, q):  # noqa: F811
    emu.emu_fp_mulmod.argtypes = [C.c_uint64, f64p, u64p, C.c_size_t, f64p, u64p]
    rng = np.random.default_rng(q % 1000003)
    a = [int(v) for v in rng.integers(-(1 << 52), 1 << 52, 4000)] + [int(v) for v in rng.integers(-q, q, 4000)]
    w = [int(v) for v in rng.integers(0, q, 8000)]
    for av in (0, 1, -1, q, -q, (1 << 52), -(1 << 52), (1 << 52) - 1, 4 * q - 1):
        for wv in (0, 1, q - 1, q // 2, q // 2 + 1, q // 2 - 1, q // 3):
            if abs(av) <= 1 << 52:
                a.append(av)
                w.append(wv)
    x, y = np.array(a, np.float64), np.array(w, np.uint64)
    out, word = np.zeros(len(a)), np.zeros(len(a), np.uint64)
    emu.emu_fp_mulmod(q, x, y, len(a), out, word)
    for i in range(len(a)):
        assert out[i] == int(out[i]) and (int(out[i]) - a[i] * w[i]) % q == 0, (a[i], w[i])
        assert 8 * abs(int(out[i])) <= 5 * q, (a[i], w[i])
        assert int(word[i]) == a[i] * w[i] % q


@pytest.mark.parametrize("q", [12289, _prime(1 << 27, 1 << 15), _prime(1 << 42, 1 << 15), _prime(1 << 50, 1 << 15)])
def test_reduce_over_its_whole_domain(emu, q):  # noqa: F811
    """fp::reduce is a representative within q / 2 + 1 for every |x| <= 2^53: at random, next to multiples of q
    and half-way between them, from the smallest NTT modulus (2^39 q and more) up."""
    emu.emu_fp_reduce.argtypes = [C.c_uint64, f64p, C.c_size_t, f64p]
    rng = np.random.default_rng(q % 1000003)
    top = (1 << 53) // q
    x = [int(v) for v in rng.integers(-(1 << 53), 1 << 53, 4000)]
    for k in [0, 1, top - 1, top // 2] + [int(v) for v in rng.integers(0, top, 500)]:
        x += [s * (k * q + d) for s in (1, -1) for d in (0, 1, -1, q // 2, q // 2 + 1, q - 1)]
    x = [v for v in x + [1 << 53, -(1 << 53)] if abs(v) <= 1 << 53]
    out = np.zeros(len(x))
    emu.emu_fp_reduce(q, np.array(x, np.float64), len(x), out)
    for v, r in zip(x, out):
        assert r == int(r) and (int(r) - v) % q == 0 and 2 * abs(int(r)) <= q + 2, v


@pytest.mark.parametrize("q", [_prime(1 << 42, 1 << 15), 274876334081, 12289, _prime(1 << 61, 1 << 15), _prime(1 << 62, 1 << 15)])
@pytest.mark.parametrize("n", [1, 3, 32, 33, 500])
def test_sums_of_products(emu, q, n):  # noqa: F811
    """Long sums of products (exact FP64 sums carried over every 32 terms, 128-bit integer sums folded
    on the way) with words up to 2 q - 1 times words up to q - 1, at their largest and at random."""
    emu.emu_mont_sums.argtypes = [C.c_uint64, u64p, u64p, C.c_size_t, u64p]
    rng = np.random.default_rng(n)
    out = np.zeros(2, np.uint64)
    for x, y in ((np.full(n, 2 * q - 1, np.uint64), np.full(n, q - 1, np.uint64)),
                 (rng.integers(0, 2 * q, n, dtype=np.uint64), rng.integers(0, q, n, dtype=np.uint64)),
                 (np.zeros(n, np.uint64), np.full(n, q - 1, np.uint64))):
        emu.emu_mont_sums(q, x, y, n, out)
        want = sum(int(a) * int(b) for a, b in zip(x, y)) * pow(1 << 64, -1, q) % q
        assert [int(v) for v in out] == [want, want]


@pytest.mark.parametrize("q", [_prime(1 << 27, 1 << 14), _prime(1 << 38, 1 << 15), _prime(1 << 42, 1 << 15), _prime(1 << 42, 1 << 15, 1)])
def test_tensor_takes_words_of_any_size(emu, q):  # noqa: F811
    """The tensor's FP64 products give the words of the Barrett products for residues (0, 1, q - 1 and
    zero products among them), for words in [q, 2 q), and for larger ones, which have to go through
    the words: beyond a few q the FP64 quotient no longer fits its rounding."""
    emu.emu_tensor.argtypes = [C.c_uint64] + [u64p] * 4 + [C.c_size_t] + [u64p] * 2
    emu.emu_tensor.restype = C.c_size_t
    rng = np.random.default_rng(q % 1000003)
    edge = [0, 1, q // 2, q - 1, q, q + 1, 2 * q - 1, 2 * q, 3 * q, 4 * q - 1, 4 * q, 1 << 40, (1 << 43) - 1, 1 << 43, (1 << 52) + 5, (1 << 64) - 1]
    pairs = np.array([(a, b, c, d) for a in edge for b in edge for c in edge for d in (0, q - 1, 2 * q - 1, (1 << 43) - 1)], np.uint64)
    blocks = [pairs] + [rng.integers(0, hi, (4000, 4), dtype=np.uint64) for hi in (q, 2 * q, 1 << 40, 1 << 43, 1 << 63)]
    for k, v in enumerate(blocks):
        xa, xb, ya, yb = (np.ascontiguousarray(v[:, i]) for i in range(4))
        out, ref = np.zeros(3 * len(v), np.uint64), np.zeros(3 * len(v), np.uint64)
        taken = emu.emu_tensor(q, xa, xb, ya, yb, len(v), out, ref)
        assert (out == ref).all(), k
        if k in (1, 2):  # words below 2 q
            assert taken >= 3990 if q < 1 << 42 else taken == 0
        for i in rng.integers(0, len(v), 200):
            a, b, c, d = (int(w) for w in v[i])
            assert [int(w) % q for w in out[3 * i:3 * i + 3]] == [a * c % q, b * d % q, (a * d + b * c) % q]


def _extreme_polys(q, N, rng):
    """Residue polynomials that drive the lazy sums to their bounds, with words up to 4q - 1."""
    top = np.full(N, q - 1, np.uint64)
    alt = top.copy()
    alt[::2] = 0
    wide = rng.integers(0, 4 * q, N, dtype=np.uint64)
    return [top, alt, rng.integers(0, q, N, dtype=np.uint64), wide, np.full(N, 4 * q - 1, np.uint64)]


@pytest.mark.parametrize("logN", [10, 15, 16])
@pytest.mark.parametrize("geometry", [0, 3])
def test_emulated_transforms_at_the_edges(oracle_mod, emu, logN, geometry):  # noqa: F811
    N = 1 << logN
    q = np.array(_edges(N), np.uint64)
    p = np.array([_prime(1 << 60, N)], np.uint64)
    o = oracle_mod.OracleCtx(N, q, p, 1)
    h = emu.emu_create(N, q, len(q), p, 1, 1)
    emu.emu_set_ntt_geometry(geometry)
    try:
        rng = np.random.default_rng(logN)
        polys = [_extreme_polys(int(m), N, rng) for m in q]
        for k in range(5):
            x = np.concatenate([pl[k] for pl in polys])
            canon = x % np.repeat(q, N)
            y = x.copy()
            emu.emu_ntt(h, y, len(q), 0, 0, 0)
            want = o.ntt(canon)
            assert (y == want).all(), k
            emu.emu_ntt(h, y, len(q), 0, 0, 1)
            assert (y == canon).all(), k
            # the forward transform takes words far above 4 q of a lazily reduced modulus
            if k == 2:
                y = rng.integers(0, 1 << 63, x.size, dtype=np.uint64)
                want = o.ntt(y % np.repeat(q, N))
                emu.emu_ntt(h, y, len(q), 0, 0, 0)
                assert (y == want).all()
            y = canon.copy()
            emu.emu_ntt(h, y, len(q), 0, 0, 1)
            emu.emu_ntt(h, y, len(q), 0, 0, 0)
            assert (y == canon).all(), k
    finally:
        emu.emu_set_ntt_geometry(0)
        emu.emu_destroy(h)


@pytest.mark.parametrize("logN", [10, 11, 12, 13, 14])
def test_emulated_whole_transforms(oracle_mod, emu, logN):  # noqa: F811
    """The one-launch transform (1 to 8 CTAs a cluster) in each arithmetic: FP64 with and without
    reductions inside, lazy words and fully reduced words."""
    N = 1 << logN
    q = np.array([_prime(1 << 50, N), _prime(1 << 38, N), _prime(1 << 55, N), _prime(1 << 61, N)], np.uint64)
    o = oracle_mod.OracleCtx(N, q[:3], q[3:], 1)
    h = emu.emu_create(N, q[:3].copy(), 3, q[3:].copy(), 1, 1)
    emu.emu_ntt_whole.argtypes = emu.emu_ntt.argtypes
    try:
        for basis, mods in ((0, q[:3]), (1, q[3:])):
            x = np.concatenate([np.random.default_rng(int(m) % 1000).integers(0, int(m), N, dtype=np.uint64) for m in mods])
            y = x.copy()
            emu.emu_ntt_whole(h, y, len(mods), 0, basis, 0)
            assert (y == o.ntt(x, which=basis)).all(), basis
            emu.emu_ntt_whole(h, y, len(mods), 0, basis, 1)
            assert (y == x).all(), basis
    finally:
        emu.emu_destroy(h)


def test_launch_rules(emu):  # noqa: F811
    """On 148 SMs: one launch or two phases on both sides of every line, and 8 residues a thread in small
    launches whatever large ones were tuned to."""
    emu.emu_whole_launch.argtypes = [C.c_int, C.c_size_t, C.c_int, C.c_int]
    emu.emu_launch_geometry.argtypes = [C.c_int, C.c_int, C.c_size_t, C.c_int, C.c_int]
    whole = lambda logN, n, words: emu.emu_whole_launch(logN, n, 148, words)
    assert all(whole(logN, n, words) for logN in (10, 11, 12) for n in (1, 5000) for words in (0, 1))
    assert all(whole(13, 128, words) and not whole(13, 129, words) and not whole(15, 1, words) for words in (0, 1))
    assert [n for n in range(1, 80) if whole(14, n, 0)] == list(range(1, 65))
    assert [n for n in range(1, 80) if whole(14, n, 1)] == list(range(1, 13)) + list(range(19, 49))
    tuned = lambda words, cols, ctas: [emu.emu_launch_geometry(v, cols, ctas * 2048, 148, words) for v in range(4)]
    for words in (0, 1):
        for cols in (0, 1):
            line = 148 * (3 if words and not cols else 2)
            assert tuned(words, cols, line) == [0, 1, 0, 1] and tuned(words, cols, line + 1) == [0, 1, 2, 3]


# digits of eight 50-bit limbs over nine 50-bit P limbs (the sums' bound, every width of the ModDown);
# digits and P limbs that mix FP64 and word moduli in both roles
MIXED = [dict(logN=10, q_bits=[50] * 8, p_bits=[50] * 9, dnum=1),
         dict(logN=10, q_bits=[50, 61, 42, 55, 38, 61, 50], p_bits=[61, 50, 58, 38, 60], dnum=2),
         dict(logN=11, q_bits=[31, 27, 30, 50], p_bits=[32, 50], dnum=4)]


@pytest.mark.parametrize("prm", MIXED)
def test_emulated_mixed_key_switches(oracle_mod, emu, prm):  # noqa: F811
    O, N = oracle_mod, 1 << prm["logN"]
    p, q = O.find_primes(prm["p_bits"], prm["q_bits"], N)
    o = O.OracleCtx(N, q, p, prm["dnum"])
    h = emu.emu_create(N, q, len(q), p, len(p), prm["dnum"])
    try:
        L = len(q)
        rk = o.rotation_key(o.ternary(64, 3), 3, 11)
        for fused in (0, 1, 2):  # 2: each job's outputs divided over two blocks
            emu.emu_set_keyswitch_fusion(fused)
            for level in (L - 1, L // 2, 1):
                b, a = o.uniform(level + 1, 9), o.uniform(level + 1, 10)
                ob, oa = o.rotate(level, b, a, rk, 3)
                eb, ea = b.copy(), a.copy()
                emu.emu_keyswitch(h, level, a.copy(), rk, L - 1, eb, ea, 1, 0, o.galois(3))
                assert (eb == ob).all() and (ea == oa).all(), (fused, level)
                (ref,) = o.rescale(level, [b])
                xs = b.copy()
                emu.emu_rescale(h, level, xs)
                assert (xs[: level * N] == ref).all(), (fused, level)
    finally:
        emu.emu_set_keyswitch_fusion(0)
        emu.emu_destroy(h)


def test_emulated_rescale_of_unreduced_words(oracle_mod, emu):  # noqa: F811
    """The limbs a rescale keeps may hold words of any size (only the dropped one is transformed): both
    sequences give the rescale of their residues."""
    N = 1 << 10
    q = np.array([_prime(1 << 27, N), _prime(1 << 42, N), _prime(1 << 50, N), _prime(1 << 50, N, 1), _prime(1 << 36, N)], np.uint64)
    p = np.array([_prime(1 << 60, N)], np.uint64)
    o = oracle_mod.OracleCtx(N, q, p, 1)
    h = emu.emu_create(N, q, len(q), p, 1, 1)
    try:
        rng = np.random.default_rng(8)
        qs = np.repeat(q[:4], N)
        for hi in (1 << 51, 1 << 52, 1 << 63):
            kept = rng.integers(0, hi, 4 * N, dtype=np.uint64)
            kept[::7] = hi - 1
            kept[1::7] = qs[1::7] * (hi // qs[1::7]) - 1
            drop = rng.integers(0, int(q[4]), N, dtype=np.uint64)
            (want,) = o.rescale(4, [np.concatenate([kept % qs, drop])])
            for fused in (0, 1):
                emu.emu_set_keyswitch_fusion(fused)
                x = np.concatenate([kept, drop])
                emu.emu_rescale(h, 4, x)
                assert (x[: 4 * N] == want).all(), (hi, fused)
    finally:
        emu.emu_set_keyswitch_fusion(0)
        emu.emu_destroy(h)


@pytest.mark.parametrize("q", [_prime(1 << 42, 1 << 15), _prime(1 << 42, 1 << 15, 1), 12289, _prime(1 << 55, 1 << 15, 1)])
def test_walsh_products_at_the_edges(emu, q):  # noqa: F811
    """The Walsh products on both sides of the FP64 limit, at a small modulus (coefficients and signs
    up to 12 bits wrap) and just above the limit of the one-word sums."""
    _walsh_exact(emu, q)


@pytest.mark.gpu
@pytest.mark.parametrize("logN", [10, 11, 12, 13, 14, 15, 16])
def test_transforms_at_the_edges(wg, oracle_mod, logN):
    import torch

    N = 1 << logN
    q = np.array(_edges(N), np.uint64)
    p = np.array([_prime(1 << 60, N)], np.uint64)
    o, ctx = oracle_mod.OracleCtx(N, q, p, 1), wg.Context(N, q, p, 1)
    rng = np.random.default_rng(logN)
    polys = [_extreme_polys(int(m), N, rng) for m in q]
    for geometry in range(-1, 4):  # -1: unpinned (the one-launch transform up to 2^14)
        for d in range(2):
            for ph in range(2):
                ctx.set_ntt_geometry(d, ph, geometry)
        for k in range(5):
            x = np.concatenate([pl[k] for pl in polys])
            canon = x % np.repeat(q, N)
            dx = wg.to_device(x)
            ctx.ntt_forward(dx, len(q))
            torch.cuda.synchronize()
            assert (wg.to_host(dx) == o.ntt(canon)).all(), (geometry, k)
            ctx.ntt_inverse(dx, len(q))
            dy = wg.to_device(canon)
            ctx.ntt_inverse(dy, len(q))
            ctx.ntt_forward(dy, len(q))
            torch.cuda.synchronize()
            assert (wg.to_host(dx) == canon).all() and (wg.to_host(dy) == canon).all(), (geometry, k)


@pytest.mark.gpu
@pytest.mark.parametrize("fusion", [0, 2])
@pytest.mark.parametrize("prm", MIXED)
def test_mixed_key_switches(wg, oracle_mod, prm, fusion):
    import torch

    O, N = oracle_mod, 1 << prm["logN"]
    p, q = O.find_primes(prm["p_bits"], prm["q_bits"], N)
    o, ctx = O.OracleCtx(N, q, p, prm["dnum"]), wg.Context(N, q, p, prm["dnum"])
    ctx.set_ntt_fusion(fusion)
    L = len(q)
    s = o.ternary(64, 3)
    rk, rl = o.rotation_key(s, 3, 11), o.relin_key(s, 13)
    ctx.set_key(wg.WG_KEY_ROTATION, rk, rotation=3)
    ctx.set_key(wg.WG_KEY_RELIN, rl)
    for level in (L - 1, L // 2, 1):
        n = (level + 1) * N
        b, a, c2 = o.uniform(level + 1, 9), o.uniform(level + 1, 10), o.uniform(level + 1, 12)
        db, da, dc = wg.to_device(b), wg.to_device(a), wg.to_device(c2)
        ctx.rotate(level, db, da, 3)
        ob, oa = o.rotate(level, b, a, rk, 3)
        e0, e1 = wg.to_device(b), wg.to_device(a)
        ctx.relin(level, e0, e1, dc)
        r0, r1 = o.relin(level, b, a, c2, rl)
        torch.cuda.synchronize()
        assert (wg.to_host(db) == ob).all() and (wg.to_host(da) == oa).all(), level
        assert (wg.to_host(e0)[:n] == r0).all() and (wg.to_host(e1)[:n] == r1).all(), level
        ctx.rescale(level, e0)
        (ref,) = o.rescale(level, [r0])
        torch.cuda.synchronize()
        assert (wg.to_host(e0)[: level * N] == ref).all(), level


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 7, 601])
@pytest.mark.parametrize("prm", MIXED)
def test_fused_key_products_of_many(wg, oracle_mod, prm, count):
    """The fused steps against the separate launches: one switch a job, or (601 at 2^10) two and an odd
    one left."""
    import torch

    O, N = oracle_mod, 1 << 10
    p, q = O.find_primes(prm["p_bits"], prm["q_bits"], N)
    ctx, o, L = wg.Context(N, q, p, prm["dnum"]), O.OracleCtx(N, q, p, prm["dnum"]), len(q)
    s = o.ternary(64, 3)
    ctx.set_key(wg.WG_KEY_RELIN, o.relin_key(s, 13))
    ctx.set_key(wg.WG_KEY_ROTATION, o.rotation_key(s, 3, 11), rotation=3)
    rng = np.random.default_rng(count)
    host = (rng.integers(0, 1 << 63, (4, count, L, N), dtype=np.uint64) % np.asarray(q, np.uint64)[:, None]).reshape(-1)
    levels = [1 + i % (L - 1) if i % 50 == 0 else L - 1 for i in range(count)]
    got = []
    for fusion in (0, 1):
        ctx.set_ntt_fusion(fusion)
        x = wg.to_device(host).reshape(4, count, L * N)
        ctx.batch_mul_relin_rescale_rotate(levels, list(x[0]), list(x[1]), list(x[2]), list(x[3]), [3] * count)
        torch.cuda.synchronize()
        got.append(wg.to_host(x.reshape(-1)))
    out = [g.reshape(4, count, L, N) for g in got]
    for i, level in enumerate(levels):
        assert (out[0][:2, i, :level] == out[1][:2, i, :level]).all(), i


@pytest.mark.gpu
@pytest.mark.parametrize("bits,width,fused", [(60, 4, True), (60, 5, False), (50, 12, True), (50, 13, False)])
def test_wide_base_changes_take_the_separate_launches(wg, oracle_mod, bits, width, fused):
    """Small launches fuse the base changes up to 12 sources, 4 of word moduli; launches that fill the
    device fuse them at any width.  The route shows in the launch counts, the words are the same."""
    import torch

    O, N, count = oracle_mod, 1 << 10, 160
    p, q = O.find_primes([bits] * width, [bits] * width, N)
    ctx, o = wg.Context(N, q, p, 1), O.OracleCtx(N, q, p, 1)
    s = o.ternary(64, 3)
    key = o.rotation_key(s, 3, 11)
    ctx.set_key(wg.WG_KEY_ROTATION, key, rotation=3)
    ctx.set_key(wg.WG_KEY_RELIN, o.relin_key(s, 13))
    n = width * N
    b, a = o.uniform(width, 9), o.uniform(width, 10)
    want = o.rotate(width - 1, b, a, key, 3)
    launches, batch = [], []
    for mode in (0, 1, 2):
        ctx.set_ntt_fusion(mode)
        db, da, out = wg.to_device(b), wg.to_device(a), torch.empty(2 * n, dtype=torch.int64, device="cuda")
        n0 = wg.launch_count()
        ctx.rotate_many(width - 1, db, da, [3], out)
        n1 = wg.launch_count()
        ctx.rotate(width - 1, db, da, 3)
        n2 = wg.launch_count()
        x = [wg.to_device(b).repeat(count).reshape(count, n) for _ in range(2)]
        ctx.batch_mul_relin_rescale_rotate([width - 1] * count, list(x[0]), list(x[1]), [wg.to_device(b)] * count,
                                           [wg.to_device(a)] * count, [3] * count)
        batch.append((wg.launch_count() - n2, wg.to_host(x[0][:, : n - N].reshape(-1))))
        torch.cuda.synchronize()
        launches.append((n1 - n0, n2 - n1))
        assert (wg.to_host(db) == want[0]).all() and (wg.to_host(da) == want[1]).all(), mode
        assert (wg.to_host(out) == np.concatenate(want)).all(), mode
    assert launches[0] != launches[2] and launches[1] == launches[2 if fused else 0], launches
    assert batch[1][0] == batch[2][0] < batch[0][0]
    assert (batch[1][1] == batch[0][1]).all() and (batch[2][1] == batch[0][1]).all()


@pytest.mark.gpu
def test_linear_transform_of_unreduced_words(wg, oracle_mod):
    """The b polynomial of a linear transform's input may hold words of any size (only a is transformed):
    the result is that of its residues, in every arithmetic of the giant sums."""
    import torch

    N = 1 << 10
    q = np.array([_prime(1 << 30, N), _prime(1 << 42, N), _prime(1 << 50, N), _prime(1 << 61, N)], np.uint64)
    p = np.array([_prime(1 << 60, N)], np.uint64)
    ctx, o = wg.Context(N, q, p, 2), oracle_mod.OracleCtx(N, q, p, 2)
    s = o.ternary(64, 3)
    for r in (1, 2):
        ctx.set_key(wg.WG_KEY_ROTATION, o.rotation_key(s, r, 11 + r), rotation=r)
    rng = np.random.default_rng(9)
    diags = np.concatenate([rng.integers(0, int(m), N, dtype=np.uint64) for _ in range(4) for m in (*q, *p)])
    stage = wg.LtStage(ctx, 3, [0, 1, 2, 3], diags, 2)
    b, a = o.uniform(4, 5), o.uniform(4, 6)
    room = ((1 << 63) - 1 - b) // np.repeat(q, N)
    big = b + np.repeat(q, N) * rng.integers(0, room, dtype=np.uint64)
    out = []
    for words in (b, big):
        db, da = wg.to_device(words), wg.to_device(a)
        stage.apply([db], [da])
        torch.cuda.synchronize()
        out.append((wg.to_host(db), wg.to_host(da)))
    assert (out[0][0] == out[1][0]).all() and (out[0][1] == out[1][1]).all()
