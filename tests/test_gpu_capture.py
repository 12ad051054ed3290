"""Single operations under stream capture, and the scratch that wg_ctx_reserve sets aside.

Calls outside a capture run as batches of one (job tables staged per call); under capture they run
stage by stage on the stream's workspace.  Both must give the oracle's words, at moduli on both sides
of the FP64 limit (SMALL[1]: 36 to 61 bits; SMALL[0]: FP64 Q limbs, word P limbs).
"""
import numpy as np
import pytest

from params import SMALL

pytestmark = pytest.mark.gpu


def _setup(wg, O, prm):
    N = 1 << prm["logN"]
    p, q = O.find_primes(prm["p_bits"], prm["q_bits"], N)
    o, ctx = O.OracleCtx(N, q, p, prm["dnum"]), wg.Context(N, q, p, prm["dnum"])
    s = o.ternary(64, 3)
    keys = dict(rot=o.rotation_key(s, 3, 11), conj=o.conjugation_key(s, 7), relin=o.relin_key(s, 9))
    ctx.set_key(wg.WG_KEY_ROTATION, keys["rot"], rotation=3)
    ctx.set_key(wg.WG_KEY_CONJ, keys["conj"])
    ctx.set_key(wg.WG_KEY_RELIN, keys["relin"])
    return N, o, ctx, keys


def _calls(wg, o, ctx, keys, level):
    """name -> (the call on device buffers x[0..2], the oracle's (x[0], x[1]) for the host words)."""
    n = (level + 1) * o.N
    return {
        "keyswitch": (lambda x: ctx.keyswitch(level, x[2], wg.WG_KEY_ROTATION, x[0], x[1], True, False, rotation=3),
                      lambda b, a, c: o.keyswitch(level, c, keys["rot"], b, a, 1, 0)),
        "conjugate": (lambda x: ctx.conjugate(level, x[0], x[1]), lambda b, a, c: o.conjugate(level, b, a, keys["conj"])),
        "rescale": (lambda x: ctx.rescale(level, x, npolys=2, stride=n), lambda b, a, c: o.rescale(level, [b, a])),
        "rotate": (lambda x: ctx.rotate(level, x[0], x[1], 3), lambda b, a, c: o.rotate(level, b, a, keys["rot"], 3)),
        "relin": (lambda x: ctx.relin(level, x[0], x[1], x[2]), lambda b, a, c: o.relin(level, b, a, c, keys["relin"])),
    }


@pytest.mark.parametrize("name", ["keyswitch", "conjugate", "rescale", "rotate", "relin"])
@pytest.mark.parametrize("prm", SMALL[:2])
def test_captured_operation_matches_oracle(wg, oracle_mod, prm, name):
    """A call outside the capture (for keyswitch, conjugate and rescale that alone allocates what the
    captured one needs; rotate and relin want wg_ctx_reserve), then the capture and two replays."""
    import torch

    N, o, ctx, keys = _setup(wg, oracle_mod, prm)
    level = o.nq - 1
    run, want = _calls(wg, o, ctx, keys, level)[name]
    host = [[o.uniform(level + 1, 30 + 3 * k + i) for i in range(3)] for k in range(3)]
    live = (level if name == "rescale" else level + 1) * N
    x = torch.empty((3, (level + 1) * N), dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()

    def load(k):
        for i in range(3):
            x[i].copy_(wg.to_device(host[k][i]))
        torch.cuda.synchronize()

    def check(k):
        torch.cuda.synchronize()
        wb, wa = want(*host[k])
        assert (wg.to_host(x[0])[:live] == wb[:live]).all() and (wg.to_host(x[1])[:live] == wa[:live]).all(), (name, k)

    with torch.cuda.stream(stream):
        load(0)
        if name in ("rotate", "relin"):
            ctx.reserve()
        run(x)
        check(0)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        graph.capture_begin()
        try:
            run(x)
        finally:
            graph.capture_end()
        for k in (1, 2):
            load(k)
            graph.replay()
            check(k)


def test_reserve_covers_the_single_calls(wg, oracle_mod):
    """After wg_ctx_reserve, the first keyswitch, conjugate and rescale of a stream take no more device
    memory (the kernels were loaded by the same calls on another stream)."""
    import torch

    N, o, ctx, keys = _setup(wg, oracle_mod, SMALL[1])
    level = o.nq - 1
    calls = _calls(wg, o, ctx, keys, level)
    x = torch.stack([wg.to_device(o.uniform(level + 1, 50 + i)) for i in range(3)])
    many = torch.cat([x] * 20)  # 60 polynomials: more than one pass of the scratch
    work = [calls[k][0] for k in ("keyswitch", "conjugate", "rescale")]
    work.append(lambda _: ctx.rescale(level, many, npolys=60, stride=(level + 1) * N))
    for k in range(2):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            ctx.reserve()
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            for f in work:
                f(x)
            torch.cuda.synchronize()
            if k:
                assert torch.cuda.mem_get_info()[0] == free
    (want,) = o.rescale(level, [o.uniform(level + 1, 52)])
    many.copy_(torch.cat([wg.to_device(o.uniform(level + 1, 52))] * 60).reshape(many.shape))
    ctx.rescale(level, many, npolys=60, stride=(level + 1) * N)
    torch.cuda.synchronize()
    got = wg.to_host(many.reshape(-1)).reshape(60, -1)[:, : level * N]
    assert (got == want).all()


def test_routes_of_single_calls(wg, oracle_mod):
    """Outside a capture: a key switch of one or two limbs whose base changes are too wide to fuse goes
    stage by stage (nothing is staged for it), a rescale of one or two polynomials of many word limbs too
    (six launches, not three)."""
    import torch

    N = 1 << 10
    p, q = oracle_mod.find_primes([60] * 5, [60] * 3, N)
    o, ctx = oracle_mod.OracleCtx(N, q, p, 1), wg.Context(N, q, p, 1)
    key = o.rotation_key(o.ternary(64, 3), 3, 11)
    ctx.set_key(wg.WG_KEY_ROTATION, key, rotation=3)
    for level, staged in ((0, 0), (1, 0), (2, 1)):
        x = [o.uniform(level + 1, 70 + i) for i in range(3)]
        d = [wg.to_device(v) for v in x]
        calls = wg.host_stats()["stages"]
        ctx.keyswitch(level, d[2], wg.WG_KEY_ROTATION, d[0], d[1], True, False, rotation=3)
        torch.cuda.synchronize()
        assert wg.host_stats()["stages"] - calls == staged, level
        wb, wa = o.keyswitch(level, x[2], key, x[0], x[1], 1, 0)
        assert (wg.to_host(d[0]) == wb).all() and (wg.to_host(d[1]) == wa).all(), level

    N = 1 << 15
    p, q = oracle_mod.find_primes([60], [60] * 13, N)
    o, ctx = oracle_mod.OracleCtx(N, q, p, 13), wg.Context(N, q, p, 13)
    poly = o.uniform(13, 80)
    for level, polys, launches in ((12, 2, 6), (11, 2, 3), (12, 1, 3), (12, 3, 3)):
        n = (level + 1) * N
        d = wg.to_device(poly[:n]).repeat(polys)
        n0 = wg.launch_count()
        ctx.rescale(level, d, npolys=polys, stride=n)
        torch.cuda.synchronize()
        assert wg.launch_count() - n0 == launches, (level, polys)
        (want,) = o.rescale(level, [poly[:n]])
        assert (wg.to_host(d).reshape(polys, n)[:, : level * N] == want).all(), (level, polys)


def test_more_digits_than_a_switch_takes_are_refused(wg, oracle_mod):
    """wg_keyswitch and wg_conjugate take 16 digits, outside a capture as under it."""
    import torch

    N = 1 << 10
    p, q = oracle_mod.find_primes([50], [40] * 17, N)
    o, ctx = oracle_mod.OracleCtx(N, q, p, 17), wg.Context(N, q, p, 17)
    secret = o.ternary(64, 3)
    ctx.keygen_switch_key(wg.WG_KEY_CONJ, 0, secret, seed=7)
    for level in (15, 16):
        x = [wg.to_device(o.uniform(level + 1, 90 + i)) for i in range(3)]
        calls = [lambda: ctx.keyswitch(level, x[2], wg.WG_KEY_CONJ, x[0], x[1]), lambda: ctx.conjugate(level, x[0], x[1])]
        for call in calls:
            if level == 15:
                call()
                continue
            with pytest.raises(wg.InvalidArgument):
                call()
        torch.cuda.synchronize()
