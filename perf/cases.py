"""The calls this library's users make, with the sizes they make them at.

A case is one call (or one proof) through the package's public functions, named by
its "op" and its sizes. listed() holds the fixed ones, draw() more of the same
ranges; prepare() makes the inputs on the GPU (or on the host, where the call takes
host bytes) and run() makes the call. Field elements are 64-bit words below
p = 2^64 - 2^32 + 1, held in int64 tensors.
"""
import ctypes
import hashlib
import importlib
import random

import numpy as np
import torch

P = 0xFFFFFFFF00000001
_ctx = None


def _sg():
    return importlib.import_module("stark-swarm_b200")


def _context():
    """One context for the process, as a program that proves keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = _sg().Context(0)
    return _ctx


def listed():
    return [
        # one proof's smallest unit of work: the outer rollup of a few shards (n0 = 512),
        # nothing but launches and transcript round trips
        {"name": "rollup_outer_9", "op": "rollup", "leaves": 9},
        # the 64-byte SHA-256 record proof (2 blocks, n0 = 8192): the serving path's most common job
        {"name": "sha256_proof_64B", "op": "sha256", "bytes": 64},
        # one RSA-2048 signature check (11041 columns of 32 rows, n0 = 1024)
        {"name": "rsa2048_proof_1", "op": "rsa", "records": 1},
        # one ECDSA-P256 signature check (151334 columns of 256 rows, n0 = 8192)
        {"name": "ecdsa_proof", "op": "ecdsa"},
        # one Ed25519 signature check (41519 columns of 1024 rows, n0 = 32768)
        {"name": "ed25519_proof_32B", "op": "ed25519", "bytes": 32},
        # the LDE of a record proof's trace: a two-block SHA-256 message, 756 columns
        {"name": "lde_756x256_b32", "op": "lde", "cols": 756, "log_n": 8, "blowup": 32, "shift": 1},
        # a wide trace of 1024 rows at blowup 32 (the signature AIRs' transform; a ragged column count)
        {"name": "lde_4099x1024_b32", "op": "lde", "cols": 4099, "log_n": 10, "blowup": 32, "shift": 1},
        # the headline trace: 64 columns of 2^20 rows, coset shift 7, blowup 8
        {"name": "lde_64x2p20_b8_s7", "op": "lde", "cols": 64, "log_n": 20, "blowup": 8, "shift": 7},
        # the component inverse transform of a STIR layer (six planes)
        {"name": "intt_6x2p20", "op": "ntt", "cols": 6, "log_n": 20, "inverse": True},
        # committing to the rows of a 64-column table
        {"name": "merkle_64x2p20", "op": "merkle", "cols": 64, "leaves": 1 << 20},
        # the low-degree proof of a 2^20-point quotient
        {"name": "stir_2p20", "op": "stir", "log_n": 20},
        # the SHA-256 constraints over a long message's LDE (32 blocks, 2^17 points)
        {"name": "merge_sha256_2p12_b32", "op": "merge_sha256", "log_n": 12, "blowup": 32},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(2 ** rng.uniform(np.log2(lo), np.log2(hi))))


def draw(rng):
    op = rng.choices(["rollup", "sha256", "sha512", "rsa", "ecdsa", "ed25519", "lde", "ntt", "merkle", "stir",
                      "merge_sha256"], [4, 4, 4, 2, 1, 4, 12, 8, 8, 2, 1])[0]
    if op == "rollup":  # from a few shard hashes to a shard of some thousand records
        return {"op": op, "leaves": _log_uniform(rng, 10, 4000)}
    if op in ("sha256", "sha512"):  # record bytes, up to a large record set
        return {"op": op, "bytes": rng.choice([_log_uniform(rng, 16, 4000), rng.randrange(1, 600), rng.randrange(40, 4000)])}
    if op == "rsa":
        return {"op": op, "records": _log_uniform(rng, 2, 32)}
    if op == "ecdsa":  # chains shorter than the full scalar are the AIR's own small sizes
        return {"op": op, "rows": rng.choice([32, 64, 128, 256])}
    if op == "ed25519":
        return {"op": op, "bytes": rng.randrange(0, 600)}
    if op == "lde":
        log_n = rng.randrange(4, 21)
        blowup = rng.choice([4, 8, 16, 32])
        most = max(2, min(20000, (1 << 28) // (blowup << log_n)))
        return {"op": op, "cols": _log_uniform(rng, 1, most), "log_n": log_n, "blowup": blowup,
                "shift": rng.choice([1, 7, rng.randrange(2, P)])}
    if op == "ntt":
        log_n = rng.randrange(4, 24)
        most = max(2, min(20000, (1 << 26) >> log_n))
        return {"op": op, "cols": _log_uniform(rng, 1, most), "log_n": log_n, "inverse": rng.random() < 0.5}
    if op == "merkle":  # also leaf counts that leave ragged nodes
        cols = rng.choice([1, 2, 6, 12, 18, 48, 64, _log_uniform(rng, 1, 128)])
        return {"op": op, "cols": cols, "leaves": _log_uniform(rng, 64, (1 << 26) // cols)}
    if op == "stir":
        return {"op": op, "log_n": rng.choice([*range(9, 20), 21])}
    blowup = rng.choice([4, 32])  # at least 4096 points: below, the default gate leaves the constraints out
    return {"op": op, "log_n": rng.randrange(12 - (blowup.bit_length() - 1), 12 if blowup == 32 else 15), "blowup": blowup}


# ------------------------------------------------------------------ inputs
def _field(rows, cols, seed):
    """Uniform field elements: a high word below 2^32 - 1 keeps every value below p."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    hi = torch.randint(0, (1 << 32) - 1, (rows, cols), generator=g, device="cuda", dtype=torch.int64)
    lo = torch.randint(0, 1 << 32, (rows, cols), generator=g, device="cuda", dtype=torch.int64)
    return hi.bitwise_left_shift_(32).bitwise_or_(lo)


# P-256 (affine) and edwards25519 (extended coordinates): only to make valid signatures
_P256 = 2 ** 256 - 2 ** 224 + 2 ** 192 + 2 ** 96 - 1
_P256_N = 0xFFFFFFFF00000000FFFFFFFFFFFFFFFFBCE6FAADA7179E84F3B9CAC2FC632551
_P256_G = (0x6B17D1F2E12C4247F8BCE6E563A440F277037D812DEB33A0F4A13945D898C296,
           0x4FE342E2FE1A7F9B8EE7EB4A7C0F9E162BCE33576B315ECECBB6406837BF51F5)


def _p256_add(a, b):
    if a is None or b is None:
        return a or b
    if a[0] == b[0] and (a[1] + b[1]) % _P256 == 0:
        return None
    if a == b:
        m = 3 * (a[0] * a[0] - 1) * pow(2 * a[1], -1, _P256)
    else:
        m = (b[1] - a[1]) * pow(b[0] - a[0], -1, _P256)
    x = (m * m - a[0] - b[0]) % _P256
    return x, (m * (a[0] - x) - a[1]) % _P256


def _p256_mul(k, pt):
    r = None
    while k:
        if k & 1:
            r = _p256_add(r, pt)
        pt = _p256_add(pt, pt)
        k >>= 1
    return r


def _ecdsa_signature(rng):
    digest = rng.randbytes(32)
    d, k = rng.randrange(1, _P256_N), rng.randrange(1, _P256_N)
    r = _p256_mul(k, _P256_G)[0] % _P256_N
    s = pow(k, -1, _P256_N) * (int.from_bytes(digest, "big") + r * d) % _P256_N
    return _p256_mul(d, _P256_G), r, s, digest


_ED_P = 2 ** 255 - 19
_ED_L = 2 ** 252 + 27742317777372353535851937790883648493
_ED_D = -121665 * pow(121666, -1, _ED_P) % _ED_P


def _ed_add(p, q):
    a = (p[1] - p[0]) * (q[1] - q[0]) % _ED_P
    b = (p[1] + p[0]) * (q[1] + q[0]) % _ED_P
    c = 2 * p[3] * q[3] * _ED_D % _ED_P
    d = 2 * p[2] * q[2] % _ED_P
    e, f, g, h = b - a, d - c, d + c, b + a
    return e * f % _ED_P, g * h % _ED_P, f * g % _ED_P, e * h % _ED_P


def _ed_mul(k):
    y = 4 * pow(5, -1, _ED_P) % _ED_P
    xx = (y * y - 1) * pow(_ED_D * y * y + 1, -1, _ED_P) % _ED_P
    x = pow(xx, (_ED_P + 3) // 8, _ED_P)
    if (x * x - xx) % _ED_P:
        x = x * pow(2, (_ED_P - 1) // 4, _ED_P) % _ED_P
    x = _ED_P - x if x & 1 else x
    q, r = (x, y, 1, x * y % _ED_P), (0, 1, 1, 0)
    while k:
        if k & 1:
            r = _ed_add(r, q)
        q = _ed_add(q, q)
        k >>= 1
    zi = pow(r[2], -1, _ED_P)
    x, y = r[0] * zi % _ED_P, r[1] * zi % _ED_P
    return (y | (x & 1) << 255).to_bytes(32, "little")


def _ed_signature(rng, n):
    msg, key = rng.randbytes(n), hashlib.sha512(rng.randbytes(32)).digest()
    a = int.from_bytes(key[:32], "little") & ((1 << 254) - 8) | 1 << 254
    pub = _ed_mul(a)
    r = int.from_bytes(hashlib.sha512(key[32:] + msg).digest(), "little") % _ED_L
    rb = _ed_mul(r)
    h = int.from_bytes(hashlib.sha512(rb + pub + msg).digest(), "little")
    return pub, rb + ((r + h * a) % _ED_L).to_bytes(32, "little"), msg


def _arities(leaves):
    got = []
    while leaves > 1:
        got.append(16)
        leaves = -(-leaves // 16)
    return got


def prepare(case, seed):
    sg, op, rng = _sg(), case["op"], random.Random(seed)
    s = {"op": op, "sg": sg, "ctx": _context(), "pi": rng.randbytes(32)}
    if op == "rollup":
        s["leaves"] = np.random.default_rng(seed).integers(0, P, case["leaves"], dtype=np.uint64)
    elif op in ("sha256", "sha512"):
        s["msg"] = rng.randbytes(case["bytes"])
    elif op == "rsa":
        # a 2048-bit modulus, a signature below it and the message it opens to
        n = rng.getrandbits(2048) | 1 << 2047 | 1
        sigs = [rng.randrange(n) for _ in range(case["records"])]
        s["records"] = [(n, x, pow(x, 65537, n)) for x in sigs]
    elif op == "ecdsa":
        rows = case.get("rows", 256)
        s["sig"] = _ecdsa_signature(rng)
        if rows != 256:
            s["chains"] = (_P256_G, [rng.randrange(2) for _ in range(rows)], s["sig"][0],
                           [rng.randrange(2) for _ in range(rows)])
    elif op == "ed25519":
        s["sig"] = _ed_signature(rng, case["bytes"])
    elif op == "lde":
        n = 1 << case["log_n"]
        s.update(trace=_field(case["cols"], n, seed), blowup=case["blowup"], shift=case["shift"],
                 out=torch.empty(case["cols"], n * case["blowup"], device="cuda", dtype=torch.int64))
    elif op == "ntt":
        s.update(x=_field(case["cols"], 1 << case["log_n"], seed), log_n=case["log_n"], inverse=case["inverse"])
        s["out"] = torch.empty_like(s["x"])
    elif op == "merkle":
        s.update(table=_field(case["cols"], case["leaves"], seed), arities=_arities(case["leaves"]))
    elif op == "stir":
        n0 = 1 << case["log_n"]
        s.update(f0=_field(1, n0, seed), domain=sg.FriDomain(n0), params=sg.build_params(n0, s["pi"]))
    elif op == "merge_sha256":
        n = 1 << case["log_n"]
        s.update(lde=_field(sg.SHA256_WIDTH, n * case["blowup"], seed), n=n, blowup=case["blowup"], blocks=n // 128,
                 coeffs=np.random.default_rng(seed).integers(1, P, sg.SHA256_CONSTRAINTS, dtype=np.uint64),
                 out=torch.empty(n * case["blowup"], device="cuda", dtype=torch.int64))
    else:
        raise ValueError(op)
    return s


# ------------------------------------------------------------------ the calls
def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def run(s):
    sg, ctx, op = s["sg"], s["ctx"], s["op"]
    if op == "rollup":
        return _bytes(ctx.prove_hash_rollup(s["leaves"], s["pi"]))
    if op in ("sha256", "sha512"):
        prove = ctx.prove_sha256 if op == "sha256" else ctx.prove_sha512
        proof, digest = prove(s["msg"], s["pi"])
        return _bytes(proof), _bytes(digest)
    if op == "rsa":
        return _bytes(ctx.prove_rsa2048(s["records"], s["pi"]))
    if op == "ecdsa":
        if "chains" in s:
            return _bytes(ctx.prove_p256_chains(*s["chains"], s["pi"]))
        q, r, sig, digest = s["sig"]
        return _bytes(ctx.prove_p256_ecdsa(q, r, sig, digest, sg.p256_ecdsa_pi(q[0], q[1], r, sig, digest)))
    if op == "ed25519":
        pub, sig, msg = s["sig"]
        proof, pi = ctx.prove_zsk_ksk_binding_v2(pub, sig, msg, s["pi"], s["pi"])
        return _bytes(proof), _bytes(pi)
    if op == "lde":
        return ctx.lde(s["trace"], s["blowup"], s["shift"], s["out"])
    if op == "ntt":
        return ctx.ntt(s["x"], s["log_n"], s["inverse"], s["out"])
    if op == "merkle":
        return _bytes(ctx.merkle_commit(s["table"], s["arities"], 0))
    if op == "stir":
        return _bytes(ctx.deep_fri_prove(s["f0"], s["domain"], s["params"]))
    return ctx.merge_sha256(s["lde"], s["n"], s["blowup"], s["coeffs"], s["blocks"], out=s["out"])


# ------------------------------------------------------------------ what a call cannot do without
_MUL = 8       # 32-bit multiply-adds of a field product and its reduction
_ADD = 3       # 32-bit operations of a field addition
_KECCAK = 24 * 180  # 32-bit operations of one Keccak-f[1600]


def _ntt_ops(cols, log_n):
    """log_n radix-2 levels: half a product and one addition an element and level."""
    return cols * (1 << log_n) * log_n * (_MUL / 2 + _ADD)


def _lde_ops(cols, log_n, blowup):
    return _ntt_ops(cols, log_n) * (1 + blowup)


def _leaf_ops(cols, leaves):
    return leaves * (-(-(32 + 8 * cols + 1) // 136)) * _KECCAK


def _stir_ops(log_n):
    """Leaves, inverse transform, out-of-domain sums and fold of every layer; a layer has
    six planes and an eighth of the points of the one before."""
    ops, n, planes = 0.0, log_n, 1
    while n > 0:
        ops += _ntt_ops(planes, n) + (1 << n) * planes * 5 * (_MUL + _ADD) + _leaf_ops(planes, 1 << n)
        n, planes = n - 3, 6
    return ops


def _proof_work(in_bytes, cols, log_n, blowup, products):
    """A whole proof: the trace's LDE, `products` field products a row and constraint set, and the STIR proof."""
    lg = log_n + blowup.bit_length() - 1
    return {"bytes": in_bytes + 100000, "flops": _lde_ops(cols, log_n, blowup) + (products << lg) * _MUL + _stir_ops(lg)}


def work(case):
    op = case["op"]
    if op == "rollup":
        lg = max(4, (case["leaves"] - 1).bit_length())
        return _proof_work(8 * case["leaves"], 4, lg, 32, 3)
    if op in ("sha256", "sha512"):
        width, constraints, block, pad = (756, 766, 64, 9) if op == "sha256" else (1510, 1526, 128, 17)
        blocks = -(-(case["bytes"] + pad) // block)
        return _proof_work(case["bytes"], width, max(7, (128 * blocks - 1).bit_length()), 32, constraints)
    if op == "rsa":
        return _proof_work(768 * case["records"], 11041 * case["records"], 5, 32, 24000 * case["records"])
    if op == "ecdsa":
        return _proof_work(160, 151334, case.get("rows", 256).bit_length() - 1, 32, 311000)
    if op == "ed25519":
        return _proof_work(96 + case["bytes"], 15453, 10, 32, 40000)
    n = 1 << case["log_n"] if "log_n" in case else 0
    if op == "lde":
        return {"bytes": 8 * case["cols"] * n * (1 + case["blowup"]),
                "flops": _lde_ops(case["cols"], case["log_n"], case["blowup"])}
    if op == "ntt":
        return {"bytes": 16 * case["cols"] * n, "flops": _ntt_ops(case["cols"], case["log_n"])}
    if op == "merkle":
        return {"bytes": 8 * case["cols"] * case["leaves"],
                "flops": _leaf_ops(case["cols"], case["leaves"]) + case["leaves"] / 15 * 5 * _KECCAK}
    if op == "stir":
        return {"bytes": 8 * n, "flops": _stir_ops(case["log_n"])}
    points = n * case["blowup"]
    return {"bytes": 8 * points * 757, "flops": points * 4 * 766 * _MUL + 2 * _ntt_ops(1, case["log_n"] + 5)}


# ------------------------------------------------------------------ transforms in plain numpy
def _mulmod(a, b):
    m, s = np.uint64(0xFFFFFFFF), np.uint64(32)
    a0, a1, b0, b1 = a & m, a >> s, b & m, b >> s
    t = a0 * b0
    u = a1 * b0 + (t >> s)
    v = a0 * b1 + (u & m)
    lo, hi = (t & m) | v << s, a1 * b1 + (u >> s) + (v >> s)
    h0, h1 = hi & m, hi >> s  # 2^64 = 2^32 - 1 and 2^96 = -1
    r = np.where(lo < h1, lo - h1 - m, lo - h1)
    w = h0 * m
    x = r + w
    x = np.where(x < w, x + m, x)
    return np.where(x >= np.uint64(P), x - np.uint64(P), x)


def _addmod(a, b):
    s = a + b
    return np.where((s < a) | (s >= np.uint64(P)), s - np.uint64(P), s)


def _submod(a, b):
    d = a - b
    return np.where(a < b, d + np.uint64(P), d)


def _powers(w, n):
    out = np.ones(1, dtype=np.uint64)
    while out.size < n:
        out = np.concatenate([out, _mulmod(out, np.uint64(pow(int(w), out.size, P)))])
    return out[:n]


def _transform(x, inverse):
    """X[i] = sum_k x[k] w^(ik) over the last axis, w the generator of the 2-adic subgroup's chain from 7."""
    n = x.shape[-1]
    w = pow(7, (P - 1) >> 32, P)
    for _ in range(32 - (n.bit_length() - 1)):
        w = w * w % P
    w = pow(w, -1, P) if inverse else w
    tw, y, m = _powers(w, max(1, n // 2)), x[..., None, :], n
    while m > 1:  # (..., blocks, m) -> (..., 2 blocks, m / 2), outputs in natural order by the block index
        a, b = y[..., : m // 2], y[..., m // 2:]
        even, odd = _addmod(a, b), _mulmod(_submod(a, b), tw[:: n // m][: m // 2])
        y, m = np.concatenate([even, odd], axis=-2), m // 2
    y = y[..., 0]
    return _mulmod(y, np.uint64(pow(n, -1, P))) if inverse else y


def exact(case, seed):
    """The transforms' values, where plain numpy has them soon; the other calls return digests, proofs or
    sums of constraints that only their own definition gives."""
    op = case["op"]
    if op == "ntt" and case["cols"] << case["log_n"] <= 1 << 23:
        x = _field(case["cols"], 1 << case["log_n"], seed).cpu().numpy().view(np.uint64)
        return torch.from_numpy(_transform(x, case["inverse"]).view(np.int64))
    if op == "lde" and case["cols"] * case["blowup"] << case["log_n"] <= 1 << 23:
        n, n0 = 1 << case["log_n"], case["blowup"] << case["log_n"]
        x = _field(case["cols"], n, seed).cpu().numpy().view(np.uint64)
        c = np.zeros((case["cols"], n0), dtype=np.uint64)
        c[:, :n] = _mulmod(_transform(x, True), _powers(case["shift"], n))
        return torch.from_numpy(_transform(c, False).view(np.int64))
    return None
