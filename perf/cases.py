"""The measured work of this framework: public entry points over the ranges they are used in.

Every case is a dict of plain values; prepare() makes its device inputs from a seed together
with the context and keys a program keeps, run() is one pass. Contexts and keys are kept
between states of one case: a program generates them once and evaluates many ciphertexts.
Residues are uniform in [0, q): ciphertexts, keys and NTT-domain plaintexts are.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ccmm-rs_b200"))  # the package of the tree this is run from

import ckks_b200 as cb  # noqa: E402
from ckks_b200 import fft2  # noqa: E402
from ckks_b200.params import chain  # noqa: E402


def listed():
    return [
        # one ciphertext of the N = 4096 multiplication chain into the NTT domain: the smallest call
        {"name": "ntt_one_ct", "kind": "ntt", "log_n": 12, "limbs": 3, "bits": "mixed", "polys": 2, "inverse": False},
        # the batched transform workload: 64 polynomials of 32 limbs, there and back
        {"name": "ntt_batch", "kind": "ntt", "log_n": 16, "limbs": 32, "bits": "50", "polys": 64, "inverse": True},
        # 60-bit primes (the integer networks) in a ragged batch
        {"name": "ntt_60bit", "kind": "ntt", "log_n": 13, "limbs": 5, "bits": "60", "polys": 9, "inverse": True},
        # the N = 4096 chain: multiply, relinearize, rescale, rotate by one, a batch of pairs
        {"name": "chain_n12", "kind": "multiply", "log_n": 12, "limbs": 3, "bits": "mixed", "aux": 1, "base_log": 20,
         "pairs": 64, "rotate": True},
        # an ordinary product at depth: few pairs at the matrix product's ring
        {"name": "multiply_n15", "kind": "multiply", "log_n": 15, "limbs": 14, "bits": "50", "aux": 2, "base_log": 20,
         "pairs": 3, "rotate": False},
        # one rotation of one ciphertext at the rotation workload's ring: latency of a single key switch
        {"name": "rotate_one", "kind": "rotate", "log_n": 16, "limbs": 24, "bits": "50", "aux": 3, "base_log": 32,
         "cts": 1},
        # the rotation workload: hoisted rotations of a batch of ciphertexts
        {"name": "hoisted_16x16", "kind": "hoisted", "log_n": 16, "limbs": 24, "bits": "50", "aux": 3, "base_log": 32,
         "cts": 16, "keys": 16},
        # one radix-4 stage of the encrypted 256 x 256 FFT over eight images (two ciphertexts each)
        {"name": "stage_16x6", "kind": "stage", "log_n": 16, "limbs": 24, "bits": "50", "aux": 3, "base_log": 32,
         "cts": 16, "keys": 6},
        # a whole encrypted 64 x 64 FFT of three images: six stages of small launches
        {"name": "fft2_64", "kind": "fft2", "limbs": 8, "bits": "50", "aux": 3, "base_log": 32, "images": 3},
        # the structured encrypted matrix product, d = 32
        {"name": "ccmm_32", "kind": "ccmm", "log_n": 15, "limbs": 14, "bits": "50", "aux": 2, "base_log": 20, "m": 32,
         "k": 32, "n": 32},
        # the modular plaintext matrix product at its benchmarked size and 35-bit modulus
        {"name": "park_4096", "kind": "park", "rows": 4096, "inner": 4096, "cols": 4096, "modulus": 0x7ffff6001},
        # encode and decode of a few messages at the rotation workload's ring
        {"name": "codec_n16", "kind": "codec", "log_n": 16, "limbs": 24, "bits": "50", "messages": 4, "log_scale": 50},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ntt", "ntt", "multiply", "rotate", "hoisted", "hoisted", "stage", "fft2", "ccmm", "park", "park",
                       "codec"])
    if kind == "ntt":
        c = {"kind": kind, "log_n": rng.randint(12, 16), "limbs": _log_int(rng, 1, 32),
             "bits": rng.choice(["40", "50", "50", "60"]), "polys": _log_int(rng, 1, 64), "inverse": rng.random() < 0.5}
    elif kind == "multiply":
        mixed = rng.random() < 0.3
        c = {"kind": kind, "log_n": rng.randint(12, 15), "limbs": 3 if mixed else rng.randint(2, 14),
             "bits": "mixed" if mixed else "50", "aux": rng.randint(1, 2), "base_log": 20,
             "pairs": _log_int(rng, 1, 64), "rotate": rng.random() < 0.5}
        while c["pairs"] * c["limbs"] ** 2 << c["log_n"] > 1 << 27:
            c["pairs"] = max(1, c["pairs"] // 2)
            c["log_n"] -= c["pairs"] == 1
    elif kind in ("rotate", "hoisted", "stage"):
        c = {"kind": kind, "log_n": rng.randint(12, 16), "limbs": rng.randint(3, 24), "bits": "50",
             "aux": rng.randint(1, 3), "base_log": rng.choice([20, 32, 32]), "cts": _log_int(rng, 1, 16)}
        if kind != "rotate":
            c["keys"] = _log_int(rng, 1, 32 if kind == "hoisted" else 8)
        # key bytes and output bytes stay within the listed batch's
        while _key_words(c) * c.get("keys", 1) > 2.1e9 or c["cts"] * c.get("keys", 1) > 256:
            c["keys"] = max(1, c["keys"] // 2)
    elif kind == "fft2":
        c = {"kind": kind, "limbs": rng.randint(7, 12), "bits": "50", "aux": rng.randint(1, 3),
             "base_log": rng.choice([20, 32]), "images": _log_int(rng, 1, 8)}
    elif kind == "ccmm":
        c = {"kind": kind, "log_n": rng.randint(12, 15), "limbs": rng.randint(2, 14), "bits": "50", "aux": 1,
             "base_log": 20, "m": _log_int(rng, 1, 48), "k": _log_int(rng, 1, 48), "n": _log_int(rng, 1, 48)}
        while c["m"] * c["n"] > 1024 or c["m"] * c["k"] + c["k"] * c["n"] > 2048:
            c["m"], c["k"], c["n"] = [max(1, (3 * x) // 4) for x in (c["m"], c["k"], c["n"])]
    elif kind == "park":
        c = {"kind": kind, "rows": _log_int(rng, 1, 4096), "inner": _log_int(rng, 1, 4096),
             "cols": _log_int(rng, 1, 4096), "modulus": rng.randrange(1 << rng.randint(6, 61), 1 << 62) | 1}
        bits = rng.randint(8, 62)
        c["modulus"] = (c["modulus"] >> (62 - bits)) | 1 | 1 << (bits - 1)
        if bits > 40:  # wider moduli cost up to 2.6 times as much a product
            c["inner"] = min(c["inner"], 1500)
    else:
        c = {"kind": kind, "log_n": rng.randint(12, 16), "limbs": rng.randint(2, 24), "bits": "50",
             "messages": _log_int(rng, 1, 8), "log_scale": rng.choice([40, 45, 50])}
    return c


# ------------------------------------------------------------------ contexts, keys, inputs
def _q_bits(case):
    if case["bits"] == "mixed":  # a wide first limb, then scale primes
        return (60,) + (40,) * (case["limbs"] - 1)
    return (int(case["bits"]),) * case["limbs"]


def _log_n(case):
    return case.get("log_n", 12)  # a 64 x 64 image packs into N = 4096


def _log_q(case):
    return sum(_q_bits(case))


def _digits(case, limbs=None):
    bits = sum(_q_bits(case)[:limbs])
    return -(-(bits + 1) // case["base_log"])


def _key_words(case):
    return _digits(case) * (case["limbs"] + case["aux"]) * 2 << _log_n(case)


@functools.lru_cache(maxsize=2)
def _context(log_n, q_bits, aux):
    q, p = chain(1 << log_n, q_bits, (60,) * aux)
    return cb.Context(log_n, q, p)


def _ctx(case):
    return _context(_log_n(case), _q_bits(case), case.get("aux", 0))


def _secret(n):
    return np.random.default_rng(20).integers(-1, 2, n).astype(np.int8)


@functools.lru_cache(maxsize=1)
def _keys(items):
    """The keys that a program keeps for this case (one case's at a time)."""
    case = dict(items)
    ctx, L, base = _ctx(case), case["limbs"], case["base_log"]
    s = _secret(ctx.n)
    if case["kind"] == "multiply":
        rot = cb.KeySwitchKey.hybrid_generate(ctx, L - 1, base, ctx.rotation_exponent_left(1), s, seed=11) \
            if case["rotate"] else None
        return cb.KeySwitchKey.relin_generate(ctx, L, base, s, seed=10), rot
    if case["kind"] == "ccmm":
        return cb.KeySwitchKey.relin_generate(ctx, L, base, s, seed=10)
    if case["kind"] == "fft2":
        return fft2.Fft2Plan(ctx, 64, L, s, base_log=base)
    # left rotations by 1, 2, 3, ..: the rotation workload's steps
    return [cb.KeySwitchKey.hybrid_generate(ctx, L, base, ctx.rotation_exponent_left(i + 1), s, seed=100 + i)
            for i in range(case.get("keys", 1))]


def _residues(gen, moduli, n, *lead):
    out = torch.empty(lead + (len(moduli), n), dtype=torch.int64, device="cuda")
    for i, q in enumerate(moduli):
        out[..., i, :].random_(0, q, generator=gen)
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "park":
        q = case["modulus"]
        shapes = ((case["rows"], case["inner"]), (case["inner"], case["cols"]))
        a, b = (torch.empty(s, dtype=torch.int64, device="cuda").random_(0, q, generator=gen) for s in shapes)
        return {"kind": kind, "a": a, "b": b, "q": q}
    ctx = _ctx(case)
    L, n = case["limbs"], ctx.n
    st = {"kind": kind, "ctx": ctx}
    if kind == "ntt":
        st["x"] = _residues(gen, ctx.q, n, case["polys"])
        st["y"], st["z"] = torch.empty_like(st["x"]), torch.empty_like(st["x"]) if case["inverse"] else None
        return st
    if kind == "codec":
        g = np.random.default_rng(seed)
        st["slots"] = torch.from_numpy(_slots(g, case)).cuda()
        st["limbs"], st["scale"] = L, 2.0 ** case["log_scale"]
        return st
    st["keys"] = _keys(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "cts", "pairs", "images"))))
    if kind == "multiply":
        st["a"], st["b"] = (_residues(gen, ctx.q, n, case["pairs"], 2) for _ in range(2))
    elif kind == "ccmm":
        m, k, nn = case["m"], case["k"], case["n"]
        st["a"], st["b"] = _residues(gen, ctx.q, n, k, m, 2), _residues(gen, ctx.q, n, nn, k, 2)
        st["dims"] = (m, k, nn)
    elif kind == "fft2":
        st["ct"] = _residues(gen, ctx.q, n, case["images"], 2, 2)
    else:
        st["ct"] = _residues(gen, ctx.q, n, case["cts"], 2)
        if kind == "stage":
            st["diag"] = _residues(gen, ctx.q, n, case["keys"] + 1)
    return st


def _slots(g, case):
    shape = (case["messages"], 1 << (case["log_n"] - 1))
    return g.standard_normal(shape) + 1j * g.standard_normal(shape)


def run(st):
    kind = st["kind"]
    if kind == "park":
        return cb.park_mod_pp_mm(st["a"], st["b"], st["q"])
    ctx = st["ctx"]
    if kind == "ntt":
        y = ctx.ntt_forward(st["x"], out=st["y"])
        return (y, ctx.ntt_inverse(y, out=st["z"])) if st["z"] is not None else y
    if kind == "multiply":
        relin, rot = st["keys"]
        prod = cb.multiply_relinearize_rescale(ctx, relin, st["a"], st["b"])
        return (prod, cb.rotate(ctx, rot, prod)) if rot is not None else prod
    if kind == "rotate":
        return cb.rotate(ctx, st["keys"][0], st["ct"])
    if kind == "hoisted":
        return cb.rotate_hoisted(ctx, st["keys"], st["ct"])
    if kind == "stage":
        return cb.fft_stage(ctx, st["keys"], st["diag"], st["ct"])
    if kind == "fft2":
        return st["keys"].apply(st["ct"])
    if kind == "ccmm":
        return cb.matmul_structured(ctx, st["keys"], st["a"], st["b"], *st["dims"])
    poly = cb.encode(ctx, st["slots"], st["limbs"], st["scale"])
    return poly, cb.decode(ctx, poly, st["scale"])


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: operands and keys read once, results written once. flops: two per modular
    multiply-add where the path is a contraction that no algorithm here avoids."""
    kind = case["kind"]
    if kind == "park":
        m, k, n = case["rows"], case["inner"], case["cols"]
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    n, L = 1 << _log_n(case), case["limbs"]
    poly = 8 * L * n
    if kind == "ntt":
        return {"bytes": (4 if case["inverse"] else 2) * poly * case["polys"], "flops": 0}
    if kind == "codec":
        return {"bytes": case["messages"] * (2 * poly + 16 * n), "flops": 0}
    ct = 2 * poly
    ct_out = 2 * 8 * (L - 1) * n
    relin_key = 8 * _digits(case) * 2 * L * n
    if kind == "multiply":
        b = case["pairs"] * (2 * ct + ct_out) + relin_key
        if case["rotate"]:
            b += case["pairs"] * ct_out + 8 * _digits(case, L - 1) * (L - 1 + case["aux"]) * 2 * n
        return {"bytes": b, "flops": 0}
    if kind == "ccmm":
        m, k, nn = case["m"], case["k"], case["n"]
        return {"bytes": ct * (m * k + k * nn) + ct_out * m * nn + relin_key, "flops": 2 * 4 * m * k * nn * L * n}
    if kind == "fft2":
        c = dict(case, log_n=12)
        b, images = 0, 2 * case["images"]
        for stage in range(6):
            level = L - stage
            key = 8 * _key_words(dict(c, limbs=level))
            b += (1 if stage == 5 else 6) * key + (8 if stage == 5 else 7) * 8 * level * n
        return {"bytes": b + images * (ct + 2 * 8 * (L - 6) * n), "flops": 0}
    key = 8 * _key_words(case)
    if kind == "rotate":
        return {"bytes": key + 2 * case["cts"] * ct, "flops": 0}
    macs = 2 * 2 * case["cts"] * case["keys"] * _digits(case) * (L + case["aux"]) * n
    if kind == "hoisted":
        return {"bytes": case["keys"] * key + case["cts"] * ct * (1 + case["keys"]), "flops": macs}
    return {"bytes": case["keys"] * (key + poly) + poly + case["cts"] * (ct + ct_out), "flops": macs}


def tolerance(case):
    """Canonical residues everywhere; encode and decode keep one fixed sequence of roundings."""
    return "exact"


# ------------------------------------------------------------------ 64-bit restatements
def _is_prime(v):
    d, r = v - 1, 0
    while d % 2 == 0:
        d, r = d // 2, r + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        if v % a == 0:
            return v == a
        x = pow(a, d, v)
        if x in (1, v - 1):
            continue
        for _ in range(r - 1):
            x = x * x % v
            if x == v - 1:
                break
        else:
            return False
    return True


def _primes(bits, n, count):
    got, c = [], (1 << bits) - 1
    c -= (c - 1) % (2 * n)
    while len(got) < count:
        if _is_prime(c):
            got.append(c)
        c -= 2 * n
    return got


def _moduli(case):
    bits, n = _q_bits(case), 1 << _log_n(case)
    pools = {b: iter(_primes(b, n, bits.count(b))) for b in set(bits)}
    return [next(pools[b]) for b in bits]


def _mulmod(x, y, q):
    """x y mod q for uint64 arrays below q < 2^62 (quotient from the 64-bit mantissa of long double)."""
    t = (x.astype(np.longdouble) * y / np.longdouble(q)).astype(np.uint64)
    r = (x * y - t * np.uint64(q)).astype(np.int64)
    r = np.where(r < 0, r + q, r)
    return np.where(r >= q, r - q, r).astype(np.uint64)


def _powers(base, count, q):
    p = np.ones(1, np.uint64)
    while len(p) < count:
        p = np.concatenate([p, _mulmod(p, np.uint64(pow(base, len(p), q)), q)])
    return p[:count]


def _ntt_exact(x, q, log_n):
    """[polys][N] -> entry k = poly(psi^(2k+1)): twist by psi^j, then a cyclic transform of psi^2."""
    n = 1 << log_n
    g = 2
    while pow(pow(g, (q - 1) // (2 * n), q), n, q) != q - 1:
        g += 1
    psi = pow(g, (q - 1) // (2 * n), q)
    a = _mulmod(x, _powers(psi, n, q), q)
    idx = np.array([int(format(i, "0%db" % log_n)[::-1], 2) for i in range(n)])
    a = a[:, idx]
    for s in range(1, log_n + 1):
        half = 1 << (s - 1)
        w = _powers(pow(psi, 2 * (n >> s), q), half, q)
        v = a.reshape(len(a), -1, 2, half)
        t = _mulmod(v[:, :, 1], w, q)
        u = v[:, :, 0].copy()
        v[:, :, 0] = (u + t) % np.uint64(q)
        v[:, :, 1] = (u + (np.uint64(q) - t)) % np.uint64(q)
    return a


def _park_exact(a, b, q):
    """Products of 12-bit pieces in float64 (sums below 2^53), combined modulo q in Python integers' order."""
    pieces = -(-q.bit_length() // 12)
    total = torch.zeros((a.shape[0], b.shape[1]), dtype=torch.int64, device=a.device)
    bs = [((b >> (12 * j)) & 4095).double() for j in range(pieces)]

    def shift12(v):  # 2^12 v mod q for v below q < 2^50
        return ((v << 12) % q) if q < 1 << 50 else None

    for i in reversed(range(2 * pieces - 1)):
        total = shift12(total)
        for j in range(pieces):
            if 0 <= i - j < pieces:
                p = ((a >> (12 * (i - j))) & 4095).double() @ bs[j]
                total = (total + p.to(torch.int64) % q) % q
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "ntt" and (case["polys"] * case["limbs"]) << case["log_n"] <= 1 << 19:
        st = prepare(case, seed)
        x = st["x"].cpu().numpy().view(np.uint64)
        y = np.stack([_ntt_exact(x[:, i], q, case["log_n"]) for i, q in enumerate(_moduli(case))], axis=1)
        return (y.view(np.int64), x.view(np.int64)) if case["inverse"] else y.view(np.int64)
    if kind == "park" and case["modulus"] < 1 << 50:
        st = prepare(case, seed)
        return _park_exact(st["a"], st["b"], case["modulus"])
    if kind == "codec":
        n = 1 << case["log_n"]
        idx = np.empty(n // 2, np.int64)
        e = 1
        for i in range(n // 2):
            idx[i] = (e - 1) // 2
            e = e * 5 % (2 * n)
        ev = np.zeros((case["messages"], n), np.complex128)
        s = _slots(np.random.default_rng(seed), case)
        ev[:, idx], ev[:, n - 1 - idx] = s, s.conj()
        twist = np.exp(1j * np.pi * np.arange(n) / n)
        scale = 2.0 ** case["log_scale"]
        coef = np.round((np.fft.fft(ev, axis=1) / n / twist).real * scale) / scale
        return None, (np.fft.ifft(coef * twist, axis=1) * n)[:, idx]
    return None
