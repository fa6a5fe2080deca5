"""The measured cases: what a user of this library has it do.

A case is a dict of plain values.  `prepare` makes what a server holds before
a call (a context and its plans once per process; ciphertexts, keys and
result buffers per state), `run` is the call a server makes.  Residues are
uniform modulo their primes, as those of real ciphertexts and keys are; the
parameter sets are the ones under cheddar-fhe_b200/params.

Every result is a whole residue, so every case compares exactly; `codec`
returns doubles as well, which follow a fixed operation order.
"""
import functools
import json
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cheddar-fhe_b200"))
import cheddar_b200 as chd  # noqa: E402

KS = "keyswitch_l24_a8.json"        # 24 q primes, 8 auxiliary: the key-switching set
NTT24 = "ntt_bootparam30_p24.json"  # 24 primes of the 30-bit bootstrapping set
BOOT = "bootparam_40.json"          # 47 q primes, 12 auxiliary, sparse-secret encapsulation
W64 = "bootparam_40_64bit.json"     # 26 primes of 40-55 bits, 7 of 56
KS_TOP, BOOT_TOP, W64_TOP = 22, 28, 25


def listed():
    return [
        # the smallest calls: a plaintext product and its rescale at a low level (latency, launches)
        {"name": "plain_l5", "kind": "plain", "level": 5, "engine": "default"},
        # one multiplication at the top level, as an interactive program calls it
        {"name": "hmult_l22", "kind": "hmult", "levels": "22", "engine": "default"},
        # one rotation at a middle level, the last digit ragged (14 primes in digits of 8)
        {"name": "hrot_l13", "kind": "hrot", "level": 13, "rot": 37, "engine": "default"},
        # the throughput form: a batch of independent pairs at one level, engines autotuned
        {"name": "hmult_b8", "kind": "hmult", "levels": "22,22,22,22,22,22,22,22", "engine": "auto"},
        # a server's queue: pairs at whatever level they have reached, in one call
        {"name": "hmult_mixed13", "kind": "hmult", "levels": "20,16,14,9,10,5,6,5,8,19,21,15,3", "engine": "auto"},
        # rotations of one ciphertext that share its decomposition (a convolution or a reduction tree)
        {"name": "hoist_30", "kind": "hoist", "level": 22, "rots": 30, "engine": "auto"},
        # raw transforms, one polynomial and many, forward and inverse
        {"name": "ntt_1", "kind": "ntt", "primes": 24, "count": 1},
        {"name": "ntt_32", "kind": "ntt", "primes": 24, "count": 32},
        # bootstrapping, one ciphertext per call and a batch (the largest work)
        {"name": "boot_1", "kind": "boot", "count": 1, "min_ks": False, "engine": "default"},
        {"name": "boot_b8", "kind": "boot", "count": 8, "min_ks": False, "engine": "auto"},
        # the 64-bit word path: decomposition and division back, the two halves of a key switch
        {"name": "w64_l25", "kind": "w64", "level": 25},
        # plaintexts in and out of slots, from and to host memory
        {"name": "codec_l16", "kind": "codec", "level": 16, "log_slots": 15},
    ]


def draw(rng):
    kind = rng.choice(["plain", "hmult", "hmult", "hmult", "hrot", "hrot", "hoist", "hoist", "ntt", "ntt", "boot", "w64",
                       "codec"])
    engine = rng.choice(["default", "auto"])
    if kind == "plain":
        return {"kind": kind, "level": rng.randint(1, KS_TOP), "engine": engine}
    if kind == "hmult":
        count = _log_int(rng, 1, 16)
        if rng.random() < 0.5:
            levels = [rng.randint(1, KS_TOP)] * count
        else:
            levels = [rng.randint(1, KS_TOP) for _ in range(count)]
        return {"kind": kind, "levels": ",".join(map(str, levels)), "engine": engine}
    if kind == "hrot":
        return {"kind": kind, "level": rng.randint(1, KS_TOP), "rot": rng.randint(1, (1 << 15) - 1), "engine": engine}
    if kind == "hoist":
        return {"kind": kind, "level": rng.randint(1, KS_TOP), "rots": _log_int(rng, 2, 30), "engine": engine}
    if kind == "ntt":
        return {"kind": kind, "primes": rng.randint(1, 24), "count": _log_int(rng, 1, 32)}
    if kind == "boot":
        # min-KS trades rotation keys for time: three quarters of the batch cost as much
        min_ks = rng.random() < 0.3
        return {"kind": kind, "count": _log_int(rng, 1, 5 if min_ks else 8), "min_ks": min_ks, "engine": engine}
    if kind == "w64":
        return {"kind": kind, "level": rng.randint(1, W64_TOP)}
    return {"kind": kind, "level": rng.randint(1, 16), "log_slots": rng.randint(8, 15)}


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# ------------------------------------------------------------------ contexts
# One context per parameter set and engine for the whole process, as a server
# keeps it (twiddles, level constants, compiled bootstrapping plans).

@functools.lru_cache(maxsize=None)
def _params(name):
    return json.loads(chd.load_params(name))


@functools.lru_cache(maxsize=None)
def _context(name, engine="default"):
    ctx = chd.Context.from_params(name)
    if engine == "auto":
        ctx.ks_engine = chd.BCONV_AUTO
    return ctx


@functools.lru_cache(maxsize=None)
def _context64(name):
    return chd.Context64(chd.load_params(name))


@functools.lru_cache(maxsize=None)
def _boot(engine):
    return chd.BootContext(_context(BOOT, engine))


def _shape(name):
    """(levels' prime counts, q primes in all, auxiliary primes, terminal primes)."""
    p = _params(name)
    return p["level_config"], len(p["main_primes"]) + len(p.get("terminal_primes", [])), len(p["auxiliary_primes"]), \
        len(p.get("terminal_primes", []))


class _Draw:
    """Uniform residues from one seed."""

    def __init__(self, name, seed):
        p = _params(name)
        self.primes = list(reversed(p.get("terminal_primes", []))) + p["main_primes"] + p["auxiliary_primes"]
        self.n = 1 << p["log_degree"]
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, gidx, dtype=torch.int32):
        q = torch.tensor([self.primes[int(g)] for g in gidx], dtype=dtype, device="cuda")[:, None]
        top = (1 << 31) - 1 if dtype == torch.int32 else (1 << 63) - 1
        r = torch.randint(0, top, (len(gidx), self.n), generator=self.gen, device="cuda", dtype=dtype)
        return r.remainder_(q)


def _key(ctx, draw):
    """A switching key over the whole basis."""
    beta = -(-ctx.L // ctx.alpha)
    g = list(ctx.gidx(*ctx.level_np(ctx.max_level), ctx.alpha))
    parts = [torch.stack([draw(g) for _ in range(beta)]) for _ in range(2)]
    return chd.EvaluationKey(ctx, parts[0], parts[1], on_device=True)


def _ct(ctx, draw, level, scale=1.0):
    g = ctx.gidx(*ctx.level_np(level), 0)
    parts = [draw(g), draw(g)]
    torch.cuda.synchronize()
    return ctx.import_ct(level, parts, scale=scale, on_device=True)


def _result(ctx, in_level, out_level, num_aux=0):
    """A ciphertext over its own tensor, and the part of the tensor that holds the result."""
    rows_out = ctx.num_q(out_level) + num_aux
    rows = max(ctx.num_q(in_level) + num_aux, rows_out)
    buf = torch.zeros((2, rows, ctx.n), dtype=torch.int32, device="cuda")
    ct = ctx.wrap_ct(out_level, [buf[0], buf[1]], num_aux=num_aux)
    return ct, buf[:, :rows_out]


# ----------------------------------------------------------------- the cases
def prepare(case, seed):
    state = {"kind": case["kind"]}
    {"plain": _prepare_plain, "hmult": _prepare_hmult, "hrot": _prepare_hrot, "hoist": _prepare_hoist,
     "ntt": _prepare_ntt, "boot": _prepare_boot, "w64": _prepare_w64, "codec": _prepare_codec}[case["kind"]](
        case, seed, state)
    torch.cuda.synchronize()
    return state


def run(s):
    return {"plain": _run_plain, "hmult": _run_hmult, "hrot": _run_hrot, "hoist": _run_hoist, "ntt": _run_ntt,
            "boot": _run_boot, "w64": _run_w64, "codec": _run_codec}[s["kind"]](s)


def _prepare_plain(case, seed, s):
    ctx = _context(KS, case["engine"])
    level, draw = case["level"], _Draw(KS, seed)
    s["ctx"], s["scale"] = ctx, ctx.scale(level)
    s["a"] = _ct(ctx, draw, level, s["scale"])
    s["pt"] = draw(ctx.gidx(*ctx.level_np(level), 0))
    s["tmp"], _ = _result(ctx, level, level)
    s["res"], s["out"] = _result(ctx, level, level - 1)


def _run_plain(s):
    ctx = s["ctx"]
    ctx.MultPlain(s["a"], s["pt"], s["scale"], res=s["tmp"])
    ctx.Rescale(s["tmp"], res=s["res"])
    return s["out"]


def _prepare_hmult(case, seed, s):
    ctx = _context(KS, case["engine"])
    levels, draw = [int(x) for x in case["levels"].split(",")], _Draw(KS, seed)
    s["ctx"], s["key"] = ctx, _key(ctx, draw)
    s["a"] = [_ct(ctx, draw, x) for x in levels]
    s["b"] = [_ct(ctx, draw, x) for x in levels]
    both = [_result(ctx, x, x - 1) for x in levels]
    s["res"], s["out"] = [x[0] for x in both], [x[1] for x in both]


def _run_hmult(s):
    if len(s["a"]) == 1:
        s["ctx"].HMult(s["a"][0], s["b"][0], s["key"], rescale=True, res=s["res"][0])
    else:
        s["ctx"].HMultBatch(s["a"], s["b"], s["key"], rescale=True, res_list=s["res"])
    return s["out"]


def _prepare_hrot(case, seed, s):
    ctx = _context(KS, case["engine"])
    draw = _Draw(KS, seed)
    s["ctx"], s["key"], s["rot"] = ctx, _key(ctx, draw), case["rot"]
    s["a"] = _ct(ctx, draw, case["level"])
    s["res"], s["out"] = _result(ctx, case["level"], case["level"])


def _run_hrot(s):
    s["ctx"].HRot(s["a"], s["key"], s["rot"], res=s["res"])
    return s["out"]


def _offsets(count, half=1 << 15):
    """The first `count` of +-1, +-2, +-4, ... and then 3, 5, 6, ...: distinct rotations in use order."""
    powers = [x for k in range(15) for x in ((1 << k) % half, (-(1 << k)) % half)]
    more = [x for x in range(3, 64) if x not in powers]
    return list(dict.fromkeys(powers + more))[:count]


def _prepare_hoist(case, seed, s):
    ctx = _context(KS, case["engine"])
    level, draw = case["level"], _Draw(KS, seed)
    s["ctx"], s["rots"] = ctx, _offsets(case["rots"])
    s["keys"] = [_key(ctx, draw) for _ in s["rots"]]
    s["a"] = _ct(ctx, draw, level)
    s["ext"] = [_result(ctx, level, level, ctx.alpha)[0] for _ in s["rots"]]
    both = [_result(ctx, level, level) for _ in s["rots"]]
    s["res"], s["out"] = [x[0] for x in both], [x[1] for x in both]


def _run_hoist(s):
    s["ctx"].HoistedRotate(s["a"], s["keys"], s["rots"], outs=s["ext"])
    s["ctx"].ModDownBatch(s["ext"], res_list=s["res"])
    return s["out"]


def _prepare_ntt(case, seed, s):
    ctx = _context(NTT24)
    draw = _Draw(NTT24, seed)
    s["ctx"], s["np"], s["count"] = ctx, (case["primes"], 0, 0), case["count"]
    g = list(ctx.gidx(case["primes"], 0, 0)) * case["count"]
    s["x"], s["y"] = draw(g), draw(g)


def _run_ntt(s):
    s["ctx"].ntt_raw(*s["np"], s["x"], mont=True, count=s["count"])
    s["ctx"].intt_raw(*s["np"], s["y"], mont=True, count=s["count"])
    return [s["x"], s["y"]]


def _prepare_boot(case, seed, s):
    ctx, bc = _context(BOOT, case["engine"]), _boot(case["engine"])
    draw = _Draw(BOOT, seed)
    keys = chd.EvkMap(ctx)
    keys.set_mult(_key(ctx, draw))
    keys.set_conjugation(_key(ctx, draw))
    for r in bc.rotations(min_ks=case["min_ks"]):
        keys.set_rotation(r, _key(ctx, draw))
    # sparse-secret encapsulation: one key over the lowest primes and as many
    # auxiliary ones, one of a single digit over the whole basis
    m, t = ctx.level_np(-1)
    g = list(ctx.gidx(m, t, m + t))
    keys.set_dense_to_sparse(chd.EvaluationKey(ctx, draw(g)[None], draw(g)[None], on_device=True, basis=(m, t, m + t)))
    m, t = ctx.level_np(ctx.max_level)
    g = list(ctx.gidx(m, t, ctx.alpha))
    keys.set_sparse_to_dense(chd.EvaluationKey(ctx, draw(g)[None], draw(g)[None], on_device=True,
                                               basis=(m, t, ctx.alpha)))
    s["bc"], s["keys"], s["min_ks"] = bc, keys, case["min_ks"]
    s["a"] = [_ct(ctx, draw, 0, ctx.scale(0)) for _ in range(case["count"])]
    both = [_result(ctx, ctx.max_level, bc.end_level) for _ in range(case["count"])]
    s["res"], s["out"] = [x[0] for x in both], [x[1] for x in both]


def _run_boot(s):
    if len(s["a"]) == 1:
        s["bc"].Boot(s["a"][0], s["keys"], res=s["res"][0], min_ks=s["min_ks"])
    else:
        s["bc"].BootBatch(s["a"], s["keys"], res_list=s["res"], min_ks=s["min_ks"])
    return s["out"]


def _prepare_w64(case, seed, s):
    ctx = _context64(W64)
    level, draw = case["level"], _Draw(W64, seed)
    m, t = ctx.level_np(level)
    aux = [len(_params(W64)["main_primes"]) + i for i in range(ctx.alpha)]
    beta = -(-(m + t) // ctx.alpha)
    s["ctx"], s["level"] = ctx, level
    s["src"] = draw(list(range(m + t)), torch.int64)
    s["ext"] = torch.zeros((beta, m + t + ctx.alpha, ctx.n), dtype=torch.int64, device="cuda")
    s["acc"] = torch.stack([draw(list(range(m + t)) + aux, torch.int64) for _ in range(2)])
    s["low"] = torch.zeros((2, sum(ctx.level_np(level - 1)), ctx.n), dtype=torch.int64, device="cuda")


def _run_w64(s):
    s["ctx"].modup_raw(s["level"], s["src"], s["ext"])
    s["ctx"].moddown_raw(s["level"], chd.CHD_MODDOWN_RESCALE, s["acc"], s["low"], npoly=2)
    return [s["ext"], s["low"]]


def _message(case, seed):
    rng = np.random.default_rng(seed)
    slots = 1 << case["log_slots"]
    return rng.uniform(-1, 1, slots) + 1j * rng.uniform(-1, 1, slots)


def _prepare_codec(case, seed, s):
    ctx = _context(BOOT)
    s["ctx"], s["level"], s["scale"] = ctx, case["level"], ctx.scale(case["level"])
    s["msg"] = _message(case, seed)
    s["pt"] = torch.zeros((ctx.num_q(case["level"]), ctx.n), dtype=torch.int32, device="cuda")


def _run_codec(s):
    s["ctx"].encode(s["level"], s["scale"], s["msg"], out=s["pt"])
    return [s["pt"], s["ctx"].decode(s["level"], s["scale"], s["pt"], num_slots=len(s["msg"]))]


def exact(case, seed):
    if case["kind"] != "codec":
        return None
    # decoding an encoded message gives the message, up to the integers it was rounded to
    return [None, _message(case, seed)]


def tolerance(case):
    if case["kind"] == "codec":
        # a double-precision transform over 2^15 slots in another order differs by about 1e-15 per slot
        # (the rounding to integers hides most of it), the plaintext's residues where a rounding tips over
        return {"rel": 4e-12, "max": 1e-10, "differ": 1e-4}
    return "exact"


# ------------------------------------------------------------------ the work
def work(case):
    """Bytes: each input, key and plaintext read once, each result written once.  Operations: two for every
    modular product of the transforms, base conversions and inner products that the results are made of."""
    kind = case["kind"]
    if kind == "ntt":
        limbs = 2 * case["primes"] * case["count"]
        return {"bytes": 2 * limbs * 4 * 65536, "flops": limbs * _ntt_ops()}
    if kind == "plain":
        q, lo = _num_q(KS, case["level"]), _num_q(KS, case["level"] - 1)
        return {"bytes": (3 * q + 2 * lo) * 4 * 65536,
                "flops": 2 * 2 * q * 65536 + 2 * _down_ops(q, lo)}
    if kind == "hmult":
        levels = [int(x) for x in case["levels"].split(",")]
        limbs, ops = _key_limbs(KS, max(levels)), 0
        for x in levels:
            q, lo = _num_q(KS, x), _num_q(KS, x - 1)
            limbs += 4 * q + 2 * lo
            ops += _switch_ops(KS, x) + 2 * 4 * q * 65536 + 2 * _down_ops(q + 8, lo)
        return {"bytes": limbs * 4 * 65536, "flops": ops}
    if kind in ("hrot", "hoist"):
        rots, q = case.get("rots", 1), _num_q(KS, case["level"])
        beta = -(-q // 8)
        limbs = 2 * q + rots * (_key_limbs(KS, case["level"]) + 2 * q)
        ops = _switch_ops(KS, case["level"]) + (rots - 1) * 2 * 2 * beta * (q + 8) * 65536
        return {"bytes": limbs * 4 * 65536, "flops": ops + rots * 2 * _down_ops(q + 8, q)}
    if kind == "boot":
        return _boot_work(case)
    if kind == "w64":
        p = _params(W64)
        q, lo, a = sum(p["level_config"][case["level"]]), sum(p["level_config"][case["level"] - 1]), 7
        beta = -(-q // a)
        ops = q * _ntt_ops() + beta * (q + a) * _ntt_ops() + 2 * beta * a * (q + a) * 65536
        return {"bytes": (q + beta * (q + a) + 2 * (q + a) + 2 * lo) * 8 * 65536, "flops": ops + 2 * _down_ops(q + a, lo)}
    q, slots = _num_q(BOOT, case["level"]), 1 << case["log_slots"]
    return {"bytes": 2 * q * 4 * 65536 + 2 * 16 * slots, "flops": 2 * q * _ntt_ops() + 20 * slots * case["log_slots"]}


def _num_q(name, level):
    return sum(_params(name)["level_config"][level])


def _key_limbs(name, level):
    _, _, a, ter = _shape(name)
    q, t = _num_q(name, level), _params(name)["level_config"][level][1]
    return 2 * -(-(q + ter - t) // a) * (q + a)


def _ntt_ops():
    return 2 * 65536 // 2 * 16


def _switch_ops(name, level):
    """Decomposition and inner product of one key switch."""
    _, _, a, _ = _shape(name)
    q = _num_q(name, level)
    beta = -(-q // a)
    return (q + beta * (q + a)) * _ntt_ops() + 2 * (q * (q + a) + 2 * beta * (q + a)) * 65536


def _down_ops(src, dst):
    """Division of one polynomial over `src` primes down to `dst` of them."""
    drop = max(1, src - dst)
    return (drop + dst) * _ntt_ops() + 2 * drop * dst * 65536


def _boot_work(case):
    """The seven linear transforms at their levels (splits of 8 x 4, 4 x 4 and 8 x 8 diagonals), some 30 key switches
    of EvalMod, and what is read and written whatever the order: keys, diagonals, ciphertexts."""
    a, n = 12, 65536
    levels = [(x, 8 * 4 if x == 28 else 4 * 4, 10) for x in range(28, 24, -1)] + [(x, 8 * 8, 14) for x in range(19, 16, -1)]
    # two rotation keys per transform under min-KS, 39 for all of them otherwise; multiplication and conjugation
    limbs = ((2 * 7 if case["min_ks"] else 39) + 2) * _key_limbs(BOOT, 28)
    ops = 0
    for x, diagonals, rots in levels:
        q = _num_q(BOOT, x)
        beta = -(-q // a)
        limbs += diagonals * (q + a)
        # min-KS decomposes before every rotation, hoisting once for all baby steps
        switches = rots if case["min_ks"] else 1 + rots // 2
        ops += case["count"] * (switches * _switch_ops(BOOT, x) + rots * 2 * 2 * beta * (q + a) * n +
                                2 * 2 * diagonals * (q + a) * n + rots * 2 * _down_ops(q + a, q))
    for x in range(25, 18, -1):
        q = _num_q(BOOT, x)
        ops += case["count"] * 4 * (_switch_ops(BOOT, x) + 2 * _down_ops(q + a, q))
    limbs += case["count"] * 2 * (_num_q(BOOT, 0) + _num_q(BOOT, 16))
    return {"bytes": limbs * 4 * n, "flops": ops}
