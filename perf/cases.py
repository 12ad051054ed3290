"""Cases to time this framework by: the calls that programs make, through walshgpu.

Every ciphertext is uniform residues of its chain (the work of the residue path does not depend
on the values, and every result is compared word for word); secrets, switching keys, transform
plans, the EvalMod series and encrypted key bits are real ones, made by the library as a client
and a server make them when they start.  What a program keeps for its lifetime (the context with
its keys and plans) is kept here from one `prepare` to the next for the parameter set last used;
ciphertexts, block bytes and result buffers are made anew from the seed.
"""
import os
import sys
import zlib

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aes-walsh-ckks_b200"))
import walshgpu as wg  # noqa: E402

# Parameter sets: the repository's AES presets and the rings of its primitive benchmarks and tests.
SETS = {
    "ring12": dict(logn=12, q=[50] * 7, p=[60, 60], dnum=4),
    "ring14": dict(logn=14, q=[50] * 16, p=[50] * 4, dnum=4),
    "walsh15": dict(logn=15, q=[36, 61, 42, 42] + [38] * 7 + [50, 50], p=[61] * 4, dnum=3, scale=2.0**35,
                    s2c_depth=1, s2c=[[18, 20, 23]], s2c_ratio=1, c2s=[[25, 25], [25, 25]], c2s_ratio=1, K=None,
                    degree=100, points=128, prune=1e-10),
    "xboot14": dict(logn=14, q=[31, 27, 30, 30, 30, 31, 31, 31, 31, 31, 31, 27, 27], p=[32], dnum=13),
    "xboot15": dict(logn=15, q=[38, 36, 36, 37, 37, 37] + [38] * 11, p=[38] * 5, dnum=5, scale=2.0**37, s2c_depth=2,
                    s2c=[[36], [36]], s2c_ratio=2, c2s=[[38]] * 4, c2s_ratio=1, K=12, degree=120, points=64, prune=0.0),
}


def listed():
    return [
        # one ciphertext's two polynomials to the evaluation domain: the smallest call, launches count
        dict(name="ntt_one_ct", kind="ntt", set="ring14", forward=True, polys=2, limbs=16),
        # a batch of 64 polynomials back to coefficients, larger than the L2 cache
        dict(name="ntt_batch_inverse", kind="ntt", set="walsh15", forward=False, polys=64, limbs=13),
        # single-ciphertext evaluation, one call at a time: a rotation, and a product with its relinearisation
        # and rescale at the top of the AES chain
        dict(name="rotate_one", kind="op", op="rotate", set="ring14", level=15),
        dict(name="product_one", kind="op", op="product", set="walsh15", level=12),
        # hoisted rotations of one ciphertext: the unpacking of the S-box's packed nibbles
        dict(name="rotate_many_31", kind="rotate_many", set="walsh15", level=5, rotations=31),
        # a serving batch: 64 ciphertexts at mixed levels, each product + rotation
        dict(name="batch_64", kind="batch", set="walsh15", count=64),
        # CoeffToSlot of 8 ciphertexts (a bootstrap's linear transform)
        dict(name="coeff_to_slot_8", kind="transform", set="walsh15", which="c2s", count=8),
        # one EvalMod bootstrap (latency), and a refresh's batch of XBOOT pair bootstraps
        dict(name="bootstrap_one", kind="bootstrap", set="walsh15", count=1),
        dict(name="pair_bootstrap_8", kind="pairs", set="xboot15", count=8),
        # one SubBytes layer of the XBOOT AES
        dict(name="xboot_sbox_16", kind="sbox", set="xboot15", level=5, count=16),
        # the client: encode and encrypt a batch, decrypt and decode the batch of answers
        dict(name="client_32", kind="client", set="walsh15", level=3, count=32),
        # the headline: a whole Walsh AES-CTR evaluation over 1024 counter blocks
        dict(name="aes_ctr_walsh", kind="aes", set="walsh15"),
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["ntt", "ntt", "op", "op", "rotate_many", "batch", "transform", "bootstrap", "pairs", "sbox",
                       "client"])
    if kind == "ntt":
        name = rng.choice(sorted(SETS))
        return dict(kind=kind, set=name, forward=rng.random() < 0.5, polys=_log(rng, 1, 64),
                    limbs=rng.randint(1, len(SETS[name]["q"])))
    if kind == "op":
        name = rng.choice(sorted(SETS))
        return dict(kind=kind, op=rng.choice(["rotate", "conjugate", "relin", "product"]), set=name,
                    level=rng.randint(1, len(SETS[name]["q"]) - 1))
    if kind == "rotate_many":
        name = rng.choice(["ring14", "walsh15", "xboot15"])
        return dict(kind=kind, set=name, level=rng.randint(1, len(SETS[name]["q"]) - 1), rotations=rng.randint(2, 31))
    if kind == "batch":
        return dict(kind=kind, set=rng.choice(sorted(SETS)), count=_log(rng, 1, 64), order=rng.randint(1, 1 << 20))
    if kind == "transform":
        return dict(kind=kind, set=rng.choice(["walsh15", "xboot15"]), which=rng.choice(["c2s", "s2c"]),
                    count=rng.randint(1, 8))
    if kind == "bootstrap":
        return dict(kind=kind, set=rng.choice(["walsh15", "xboot15"]), count=_log(rng, 1, 16))
    if kind == "pairs":
        return dict(kind=kind, set="xboot15", count=_log(rng, 1, 12))
    if kind == "sbox":
        return dict(kind=kind, set="xboot15", level=rng.randint(4, 6), count=_log(rng, 1, 16))
    return dict(kind=kind, set=rng.choice(["walsh15", "xboot15", "ring14"]), level=rng.randint(1, 6),
                count=_log(rng, 1, 48))


# ------------------------------------------------------------------------------------------
# what a program keeps: the context, its secrets and keys, its plans
# ------------------------------------------------------------------------------------------
class Program:
    """The context of a parameter set, with the keys, plans and key bits made on demand."""

    def __init__(self, name):
        self.name, self.spec = name, SETS[name]
        self.N = 1 << self.spec["logn"]
        p, q = wg.find_primes(self.spec["p"], self.spec["q"], self.N)
        self.ctx = wg.Context(self.N, q, p, self.spec["dnum"])
        self.L, self.K = len(q), len(p)
        rng = np.random.default_rng(zlib.crc32(name.encode()))
        self.secret, self.low = self._ternary(rng, min(256, self.N // 8)), self._ternary(rng, 32)
        self.qcol = {}
        self.made = {}

    def _ternary(self, rng, h):
        s = np.zeros(self.N, np.int8)
        s[rng.choice(self.N, h, replace=False)] = rng.choice(np.array([-1, 1], np.int8), h)
        return s

    def key(self, kind, rotation=0):
        if self.ctx.has_key(kind, rotation):
            return
        if kind in (wg.WG_KEY_DENSE_TO_SPARSE, wg.WG_KEY_SPARSE_TO_DENSE):
            src, dst = (self.secret, self.low) if kind == wg.WG_KEY_DENSE_TO_SPARSE else (self.low, self.secret)
            self.ctx.keygen_secret_switch(kind, src, dst, seed=1000 + kind)
        else:
            self.ctx.keygen_switch_key(kind, rotation, self.secret, seed=10 + kind + 16 * rotation)

    def plan(self, which):
        """The stages of a transform ("s2c", "s2c_x2" for inputs at twice the scale, "c2s") with
        their rotation keys."""
        if which not in self.made:
            s = self.spec
            q0, slots = float(self.ctx.q[0]), self.N // 2
            if which == "c2s":
                scale = np.ldexp(s["scale"], 38 - s["q"][0]) / q0 / self.bound()
                lit = wg.DftLiteral.make(True, self.L - 1, scale, scale_groups=s["c2s"], stage_count=len(s["c2s"]),
                                         active_slots=slots, log_bsgs_ratio=s["c2s_ratio"])
            else:
                scale = (q0 * 0.5) / (s["scale"] * (2.0 if which == "s2c_x2" else 1.0))
                lit = wg.DftLiteral.make(False, s["s2c_depth"], scale, scale_groups=s["s2c"],
                                         stage_count=len(s["s2c"]), active_slots=slots,
                                         log_bsgs_ratio=s["s2c_ratio"])
            stages = self.ctx.dft_plan(lit)
            for st in stages:
                idx, baby = st.download()[0], st.info()["baby"]
                for d in idx.tolist():
                    for r in (d % baby, d - d % baby):
                        if r:
                            self.key(wg.WG_KEY_ROTATION, r)
            self.made[which] = stages
        return self.made[which]

    def bound(self):
        return self.spec["K"] or wg.evalmod_k_bound(self.N, 32, -16.0)

    def bootstrap(self):
        """(parameters, SlotToCoeff, CoeffToSlot, EvalMod series) with every key a bootstrap uses."""
        if "bootstrap" not in self.made:
            s = self.spec
            params = wg.BootstrapParams(s["s2c_depth"], self.L - 1, 38, 0, self.N // 2, self.N // 2, s["scale"])
            fit = wg.evalmod_fit(self.bound(), s["degree"], 0, np.nextafter(0.25, 0.0), s["points"], s["prune"])
            for kind in (wg.WG_KEY_RELIN, wg.WG_KEY_CONJ, wg.WG_KEY_DENSE_TO_SPARSE, wg.WG_KEY_SPARSE_TO_DENSE):
                self.key(kind)
            self.made["bootstrap"] = (params, self.plan("s2c"), self.plan("c2s"), fit["coeffs"])
        return self.made["bootstrap"]

    def aes(self):
        """(key bits, scales): the 1408 encrypted round-key bits of an expanded AES key."""
        if "aes" not in self.made:
            params = self.bootstrap()[0]
            self.plan("s2c_x2")
            half = self.N // 2
            for k in range(1, 32):
                self.key(wg.WG_KEY_ROTATION, 512 * k)
                self.key(wg.WG_KEY_ROTATION, half - 512 * k)
            dev = torch.empty((1408, 2, 3 * self.N), dtype=torch.int64, device="cuda")
            bits = [(dev[k, 0], dev[k, 1]) for k in range(1408)]
            expanded = np.random.default_rng(176).integers(0, 256, 176, dtype=np.uint8).tobytes()
            scales, _ = self.ctx.aes_walsh_encrypt_round_key_bits(params, expanded, 512, self.secret, bits, seed=5)
            self.made["aes"] = (bits, scales)
        return self.made["aes"]

    def uniform(self, gen, shape, limbs, room=None):
        """Uniform residues of the first `limbs` moduli in tensors with room for `room` limbs."""
        room = room or limbs
        if limbs not in self.qcol:
            self.qcol[limbs] = torch.from_numpy(self.ctx.q[:limbs].astype(np.int64)).cuda()[:, None]
        out = torch.zeros((*shape, room, self.N), dtype=torch.int64, device="cuda")
        for i in np.ndindex(*shape):
            r = torch.randint(0, 1 << 62, (limbs, self.N), dtype=torch.int64, device="cuda", generator=gen)
            out[i][:limbs] = r % self.qcol[limbs]
        return out.view(*shape, room * self.N)


_kept = []


def _program(name):
    if not _kept or _kept[0].name != name:
        _kept[:] = []
        _kept.append(Program(name))
    return _kept[0]


def _pairs(t):
    return [(t[i, 0], t[i, 1]) for i in range(t.shape[0])]


def _slots(case, seed):
    """Slot vectors of a client batch: request bits in both parts, with the spread that answers have."""
    rng = np.random.default_rng(seed)
    shape = (case["count"], 1 << (SETS[case["set"]]["logn"] - 1))
    part = lambda: rng.integers(0, 2, shape) + 1e-3 * rng.standard_normal(shape)  # noqa: E731
    return part(), part()


def prepare(case, seed):
    pr = _program(case["set"])
    ctx, kind = pr.ctx, case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    st = {"case": dict(case), "pr": pr}
    level = case.get("level")
    if kind == "ntt":
        st["x"] = pr.uniform(gen, (case["polys"],), case["limbs"])
    elif kind == "op":
        st["x"], st["y"] = pr.uniform(gen, (2,), level + 1), pr.uniform(gen, (2,), level + 1)
        st["z"] = pr.uniform(gen, (1,), level + 1)
        {"rotate": lambda: pr.key(wg.WG_KEY_ROTATION, 1), "conjugate": lambda: pr.key(wg.WG_KEY_CONJ),
         "relin": lambda: pr.key(wg.WG_KEY_RELIN), "product": lambda: pr.key(wg.WG_KEY_RELIN)}[case["op"]]()
    elif kind == "rotate_many":
        st["x"] = pr.uniform(gen, (2,), level + 1)
        step = pr.N // 2 // 32
        st["rots"] = [step * (k + 1) for k in range(case["rotations"])]
        for r in st["rots"]:
            pr.key(wg.WG_KEY_ROTATION, r)
        st["out"] = torch.zeros((case["rotations"], 2, (level + 1) * pr.N), dtype=torch.int64, device="cuda")
    elif kind == "batch":
        rng = np.random.default_rng(case.get("order", 2026))
        n = case["count"]
        st["levels"] = rng.integers(1, pr.L, n)
        st["rots"] = [int(r) * (pr.N // 2 // 32) for r in rng.integers(1, 32, n)]
        pr.key(wg.WG_KEY_RELIN)
        for r in set(st["rots"]):
            pr.key(wg.WG_KEY_ROTATION, r)
        st["x"], st["y"] = pr.uniform(gen, (n, 2), pr.L), pr.uniform(gen, (n, 2), pr.L)
    elif kind == "transform":
        st["stages"] = pr.plan(case["which"])
        st["x"] = pr.uniform(gen, (case["count"], 2), st["stages"][0].info()["level"] + 1)
    elif kind in ("bootstrap", "pairs"):
        st["plan"] = pr.bootstrap()
        n = case["count"]
        st["x"] = pr.uniform(gen, (2 * n if kind == "pairs" else n, 2), pr.spec["s2c_depth"] + 1, pr.L)
        if kind == "bootstrap":
            st["out"] = torch.zeros((2 * n, 2, pr.L * pr.N), dtype=torch.int64, device="cuda")
    elif kind == "sbox":
        pr.key(wg.WG_KEY_RELIN)
        n = case["count"]
        st["x"] = pr.uniform(gen, (8 * n, 2), level + 1)
        st["out"] = torch.zeros((8 * n, 2, (level + 1) * pr.N), dtype=torch.int64, device="cuda")
        by8 = lambda t: [_pairs(t[8 * i: 8 * i + 8]) for i in range(n)]  # noqa: E731
        st["bits"], st["outs"] = by8(st["x"]), by8(st["out"])
    elif kind == "client":
        n, limbs = case["count"], level + 1
        st["scale"] = 2.0**35 if case["set"] == "walsh15" else 2.0**37
        st["re"], st["im"] = _slots(case, seed)
        st["seed"] = seed + 1
        st["pt"] = torch.zeros((n, limbs * pr.N), dtype=torch.int64, device="cuda")
        st["ct"] = torch.zeros((n, 2, limbs * pr.N), dtype=torch.int64, device="cuda")
        # the answers: the same slots as a server would send them, without fresh noise
        st["answer"] = torch.zeros_like(st["ct"])
        ctx.encode_slots_device(limbs, st["scale"], st["re"], st["im"], list(st["pt"]), eval_form=True)
        mask = pr.uniform(gen, (n,), limbs).cpu().numpy().view(np.uint64)
        ctx.encrypt_symmetric(level, list(st["pt"]), pr.secret, _pairs(st["answer"]), a=mask,
                              e=np.zeros((n, pr.N), np.int64))
    elif kind == "aes":
        st["plan"], (st["keys"], st["kscales"]) = pr.bootstrap(), pr.aes()
        rng = np.random.default_rng(seed)
        st["counters"], st["texts"] = (rng.integers(0, 256, 16 * 1024, dtype=np.uint8).tobytes() for _ in range(2))
        st["out"] = torch.zeros((128, 2, pr.L * pr.N), dtype=torch.int64, device="cuda")
    return st


def run(st):
    case, pr = st["case"], st["pr"]
    ctx, kind = pr.ctx, case["kind"]
    level = case.get("level")
    if kind == "ntt":
        call = ctx.ntt_forward if case["forward"] else ctx.ntt_inverse
        call(st["x"], case["limbs"], polys=case["polys"], stride=case["limbs"] * pr.N)
        return st["x"]
    if kind == "op":
        x, y, z = st["x"], st["y"], st["z"][0]
        if case["op"] == "rotate":
            ctx.rotate(level, x[0], x[1], 1)
        elif case["op"] == "conjugate":
            ctx.conjugate(level, x[0], x[1])
        elif case["op"] == "relin":
            ctx.relin(level, x[0], x[1], z)
        else:
            ctx.mul(level, x[0], x[1], y[0], y[1], z)
            ctx.relin(level, x[0], x[1], z)
            ctx.rescale(level, x, 2, (level + 1) * pr.N)
        return x
    if kind == "rotate_many":
        ctx.rotate_many(level, st["x"][0], st["x"][1], st["rots"], st["out"])
        return st["out"]
    if kind == "batch":
        x, y = st["x"], st["y"]
        ctx.batch_mul_relin_rescale_rotate(st["levels"], list(x[:, 0]), list(x[:, 1]), list(y[:, 0]), list(y[:, 1]),
                                           st["rots"])
        return x
    if kind == "transform":
        x = st["x"]
        for stage in st["stages"]:
            stage.apply(list(x[:, 0]), list(x[:, 1]))
        return x
    if kind == "bootstrap":
        x, out, n = st["x"], _pairs(st["out"]), case["count"]
        ctx.bootstrap_evalmod(*st["plan"], list(x[:, 0]), list(x[:, 1]), out[:n], out[n:])
        return st["out"]
    if kind == "pairs":
        c, n = _pairs(st["x"]), case["count"]
        params, s2c, c2s, coeffs = st["plan"]
        ctx.bootstrap_pair(params, s2c, c2s, coeffs, params.scale, list(zip(c[:n], c[n:])))
        return st["x"]
    if kind == "sbox":
        ctx.xboot_sbox(level, 2.0**37, st["bits"], st["outs"])
        return st["out"]
    if kind == "client":
        ctx.encode_slots_device(level + 1, st["scale"], st["re"], st["im"], list(st["pt"]), eval_form=True)
        ctx.encrypt_symmetric(level, list(st["pt"]), pr.secret, _pairs(st["ct"]), seed=st["seed"])
        slots = ctx.decrypt_decode(level, [st["scale"]] * case["count"], _pairs(st["answer"]), pr.secret)
        return {"ciphertexts": st["ct"], "slots": slots}
    params, s2c, c2s, coeffs = st["plan"]
    ctx.aes_ctr_walsh(params, s2c, pr.plan("s2c_x2"), c2s, coeffs, 512, 32, st["keys"], st["kscales"], 2,
                      st["counters"], st["texts"], 512, _pairs(st["out"]))
    return st["out"]


def work(case):
    """Bytes: ciphertexts in and out, and each switching key and plan diagonal a pass uses once.
    Operations (three a butterfly) for the transforms alone; elsewhere the count is the code's choice."""
    s, kind = SETS[case["set"]], case["kind"]
    N, L, K = 1 << s["logn"], len(s["q"]), len(s["p"])
    level, n = case.get("level", L - 1), case.get("count", 1)
    alpha = -(-L // s["dnum"])
    poly = lambda lv: 8.0 * N * (lv + 1)  # noqa: E731
    key = lambda lv: 8.0 * N * 2 * (lv + 1 + K) * -(-(lv + 1) // alpha)  # noqa: E731
    flops = 0.0
    if kind == "ntt":
        limbs = case["polys"] * case["limbs"]
        b, flops = 16.0 * N * limbs, 1.5 * N * s["logn"] * limbs
    elif kind == "op":
        polys = {"rotate": 4, "conjugate": 4, "relin": 5, "product": 6}[case["op"]]
        b = polys * poly(level) + key(level)
    elif kind == "rotate_many":
        b = 2 * poly(level) + case["rotations"] * (2 * poly(level) + key(level))
    elif kind == "batch":
        levels = np.random.default_rng(case.get("order", 2026)).integers(1, L, n)
        b = sum(6 * poly(int(lv)) for lv in levels) + key(L - 1) * (1 + min(31, n))
    elif kind == "transform":
        lv = L - 1 if case["which"] == "c2s" else s["s2c_depth"]
        b = 4 * n * poly(lv) + 32 * key(lv) + 64 * 8.0 * N * (lv + 1 + K)
    elif kind in ("bootstrap", "pairs"):
        b = 6 * n * poly(L - 1) + 64 * key(L - 1) + 128 * 8.0 * N * (L + K)
    elif kind == "sbox":
        b = 32 * n * poly(level) + key(level)
    elif kind == "client":
        b = 8.0 * N * n * 2 + 6 * n * poly(level)
    else:
        b = 1408 * 2 * poly(2) + 69 * key(L - 1) + 128 * 2 * poly(L - 1) + 200 * 8.0 * N * (L + K)
    return {"bytes": b, "flops": flops}


def tolerance(case):
    """Residues are whole numbers and the same word for word.  Decoded slots are 64-bit floating
    point behind an FFT of N points: 1e-13 relative covers another summation order."""
    return {"rel": 1e-13, "max": 1e-11, "differ": 0.0} if case["kind"] == "client" else "exact"


def exact(case, seed):
    """The decoded slots of a client batch: the slots encoded (rounded to whole coefficients) and
    decoded in 64 bits.  Everything else is whole numbers, compared with each other as they are."""
    if case["kind"] != "client":
        return None
    N = 1 << SETS[case["set"]]["logn"]
    scale = 2.0**35 if case["set"] == "walsh15" else 2.0**37
    re, im = _slots(case, seed)
    root = np.ones(N // 2, np.int64)  # slot j is the value at the (5^j)-th power of the 2N-th root of unity
    for j in range(1, N // 2):
        root[j] = root[j - 1] * 5 % (2 * N)
    out = np.empty((case["count"], N // 2), np.complex128)
    for k in range(case["count"]):
        spread = np.zeros(2 * N, np.complex128)
        spread[root] = re[k] + 1j * im[k]
        spread[2 * N - root] = re[k] - 1j * im[k]
        coeffs = np.rint(np.fft.fft(spread)[:N].real / N * scale)
        out[k] = np.fft.ifft(coeffs, 2 * N)[root] * (2 * N) / scale
    return {"ciphertexts": None, "slots": out}
