"""The calls that a user of libtmvpkem makes, as measurable cases.

Every case goes through the package's public entry points (tmvpkem.Context,
MixedPlan): batched key generation, encapsulation and decapsulation of the six
parameter sets from a single instance to a full batch, decapsulation with the
keys' matrices expanded beforehand and under one long-term key, a mixed-set
pass replayed as a graph, host buffers, and the raw matrix-vector product.
Buffers are device memory on the caller's stream unless the case says host.
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.getcwd(), "asfand-tmvp_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tmvpkem as T  # noqa: E402

SETS = {"lightsaber": T.LIGHTSABER, "saber": T.SABER, "firesaber": T.FIRESABER, "lightsable": T.LIGHTSABLE,
        "sable": T.SABLE, "firesable": T.FIRESABLE}
# l, log2 q, mu of each set (the key, ciphertext and expanded-matrix sizes come from the package)
SHAPE = {"lightsaber": (2, 13, 10), "saber": (3, 13, 8), "firesaber": (4, 13, 6), "lightsable": (2, 11, 2),
         "sable": (3, 11, 2), "firesable": (4, 11, 2)}
MIXED_SETS = ("lightsaber", "saber", "firesaber", "sable")
# 32-bit operations of one Keccak-f[1600]: 24 rounds of 180 three-input logic operations and funnel shifts
KECCAK_OPS = 24 * 180

_ctx = None


def _context():
    """The process's one context, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = T.Context(0)
    return _ctx


def listed():
    return [
        # one client's handshake: the latency of a single decapsulation
        {"name": "dec_saber_1", "op": "dec", "set": "saber", "n": 1},
        # a small server batch, not a power of two, of the largest module rank
        {"name": "dec_firesaber_1000", "op": "dec", "set": "firesaber", "n": 1000},
        # an odd mid-size batch of the second family
        {"name": "dec_sable_20011", "op": "dec", "set": "sable", "n": 20011},
        # the headline workload: 64K independent keys and ciphertexts
        {"name": "dec_saber_65536", "op": "dec", "set": "saber", "n": 65536},
        # a serving batch whose keys have their matrix expanded once (the serving loop's largest batch)
        {"name": "dec_cached_saber_4096", "op": "dec_cached", "set": "saber", "n": 4096},
        # a server's one long-term key, many clients
        {"name": "dec_onekey_saber_65536", "op": "dec_onekey", "set": "saber", "n": 65536},
        # interleaved requests of four sets in one captured pass, 1-8192 instances each
        {"name": "dec_mixed_24", "op": "dec_mixed", "groups": 24, "most": 8192, "pick": 11},
        # the whole call on pinned host buffers: copies in, decapsulation, keys out
        {"name": "dec_host_saber_65536", "op": "dec_host", "set": "saber", "n": 65536},
        # a few clients' encapsulations at once
        {"name": "enc_lightsaber_17", "op": "enc", "set": "lightsaber", "n": 17},
        # bulk encapsulation
        {"name": "enc_saber_65536", "op": "enc", "set": "saber", "n": 65536},
        # ephemeral key generation for many sessions
        {"name": "keypair_saber_16384", "op": "keypair", "set": "saber", "n": 16384},
        # the raw matrix-vector product: 3x3 polynomials mod 2^13, CBD(8) secrets
        {"name": "matvec_l3_16384", "op": "matvec", "l": 3, "eq": 13, "mu": 8, "transpose": False, "n": 16384},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    op = rng.choice(("dec", "dec", "dec", "dec_cached", "dec_onekey", "dec_mixed", "dec_host", "enc", "enc", "keypair",
                     "matvec"))
    if op == "dec_mixed":
        return {"op": op, "groups": rng.randint(2, 16), "most": _log_uniform(rng, 16, 8192),
                "pick": rng.randrange(1 << 20)}
    if op == "matvec":
        l, eq = rng.choice((2, 3, 4)), rng.choice((9, 11, 13))
        return {"op": op, "l": l, "eq": eq, "mu": rng.choice((2, 6, 8, 10)), "transpose": rng.random() < 0.5,
                "n": _log_uniform(rng, 1, 16384 if l < 4 else 9216)}
    name = rng.choice(sorted(SETS))
    most = {2: 65536, 3: 65536, 4: 36864}[SHAPE[name][0]]
    return {"op": op, "set": name, "n": _log_uniform(rng, 1, 4096 if op == "dec_cached" else most)}


def _groups(case):
    """The (set, count) pairs of a mixed case."""
    rng = random.Random(case["pick"])
    return [(rng.choice(MIXED_SETS), rng.randint(1, case["most"])) for _ in range(case["groups"])]


def _bytes(gen, n, width):
    return torch.randint(0, 256, (n, width), dtype=torch.uint8, device="cuda", generator=gen)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _empty(n, width):
    return torch.empty((n, width), dtype=torch.uint8, device="cuda")


def _keys(gen, set_id, n):
    z = T.sizes(set_id)
    pk, sk = _empty(n, z.pk_bytes), _empty(n, z.sk_bytes)
    _context().kem_keypair_ptr(set_id, n, pk, sk, _bytes(gen, n, 96), stream=_stream())
    return pk, sk


def _ciphertexts(gen, set_id, pk):
    """Ciphertexts for pk; one in 61 arrives damaged and takes the rejection path."""
    n, z = pk.shape[0], T.sizes(set_id)
    ct, ss = _empty(n, z.ct_bytes), _empty(n, 32)
    _context().kem_enc_ptr(set_id, n, ct, ss, pk, _bytes(gen, n, 32), stream=_stream())
    ct[60::61, 7] ^= 0x10
    return ct


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, ctx = case["op"], _context()
    if op == "dec_mixed":
        groups = []
        for name, n in _groups(case):
            pk, sk = _keys(gen, SETS[name], n)
            groups.append((SETS[name], _empty(n, 32), _ciphertexts(gen, SETS[name], pk), sk))
        torch.cuda.synchronize()
        return {"op": op, "groups": groups, "plan": T.MixedPlan(ctx, groups)}
    n = case["n"]
    if op == "matvec":
        l, half = case["l"], case["mu"] // 2
        A = torch.randint(0, 1 << case["eq"], (n, l, l, 256), dtype=torch.int16, device="cuda", generator=gen)
        bits = torch.randint(0, 2, (2, half, n, l, 256), dtype=torch.int8, device="cuda", generator=gen)
        s = (bits[0].sum(0) - bits[1].sum(0)).to(torch.int8)  # centred binomial secrets
        return {"op": op, "case": dict(case), "A": A, "s": s,
                "out": torch.empty((n, l, 256), dtype=torch.int16, device="cuda")}
    set_id = SETS[case["set"]]
    z = T.sizes(set_id)
    st = {"op": op, "set": set_id, "n": n}
    if op == "keypair":
        st.update(coins=_bytes(gen, n, 96), pk=_empty(n, z.pk_bytes), sk=_empty(n, z.sk_bytes))
    elif op == "enc":
        st.update(pk=_keys(gen, set_id, n)[0], coins=_bytes(gen, n, 32), ct=_empty(n, z.ct_bytes), ss=_empty(n, 32))
    elif op == "dec_onekey":
        pk, sk = _keys(gen, set_id, 1)
        st.update(ct=_ciphertexts(gen, set_id, pk.expand(n, -1).contiguous()), sk=sk, ss=_empty(n, 32))
    else:
        pk, sk = _keys(gen, set_id, n)
        st.update(ct=_ciphertexts(gen, set_id, pk), sk=sk, ss=_empty(n, 32))
        if op == "dec_cached":
            st["a"] = _empty(n, T.genmatrix_bytes(set_id))
            ctx.genmatrix_ptr(set_id, n, st["a"], pk, stream=_stream())
        elif op == "dec_host":
            for k in ("ct", "sk", "ss"):
                st[k] = st[k].cpu().pin_memory()
    torch.cuda.synchronize()
    return st


def run(st):
    op, ctx, s = st["op"], _context(), _stream()
    if op == "dec" or op == "dec_host":
        ctx.kem_dec_ptr(st["set"], st["n"], st["ss"], st["ct"], st["sk"], stream=s)
        return st["ss"]
    if op == "dec_cached":
        ctx.kem_dec_a_ptr(st["set"], st["n"], st["ss"], st["ct"], st["sk"], st["a"], stream=s)
        return st["ss"]
    if op == "dec_onekey":
        ctx.kem_dec_onekey_ptr(st["set"], st["n"], st["ss"], st["ct"], st["sk"], stream=s)
        return st["ss"]
    if op == "dec_mixed":
        st["plan"].launch(stream=s)
        return [g[1] for g in st["groups"]]
    if op == "enc":
        ctx.kem_enc_ptr(st["set"], st["n"], st["ct"], st["ss"], st["pk"], st["coins"], stream=s)
        return {"ct": st["ct"], "ss": st["ss"]}
    if op == "keypair":
        ctx.kem_keypair_ptr(st["set"], st["n"], st["pk"], st["sk"], st["coins"], stream=s)
        return {"pk": st["pk"], "sk": st["sk"]}
    c = st["case"]
    ctx.matvec_ptr(c["n"], c["l"], c["eq"], c["transpose"], st["out"], st["A"], st["s"], stream=s)
    return st["out"]


def _perms(nbytes, rate):
    return nbytes // rate + 1  # absorbed, the padding always taking a byte


def _squeezes(nbytes):
    return -(-nbytes // 168)


def _instance_work(op, name):
    """(bytes, operations) of one instance: its inputs read and outputs written
    once; its polynomial products as 256 x 256 Toeplitz products (2 operations
    a term) and its Keccak-f permutations."""
    l, eq, mu = SHAPE[name]
    z = T.sizes(SETS[name])
    gen_a, gen_s = _squeezes(l * l * eq * 32), _squeezes(l * mu * 32)
    h_pk, h_ct = _perms(z.pk_bytes, 136), _perms(z.ct_bytes, 136)
    if op == "keypair":
        return 96 + z.pk_bytes + z.sk_bytes, 2 * 65536 * l * l + KECCAK_OPS * (1 + gen_a + gen_s + h_pk)
    if op == "enc":
        return (32 + z.pk_bytes + z.ct_bytes + 32,
                2 * 65536 * (l * l + l) + KECCAK_OPS * (1 + h_pk + 1 + gen_s + gen_a + h_ct + 1))
    ops = 2 * 65536 * (l + l * l + l) + KECCAK_OPS * (h_ct + 1 + gen_s + 1)
    nbytes = z.ct_bytes + 32
    if op != "dec_onekey":
        nbytes += z.sk_bytes
    if op == "dec_cached":
        nbytes += T.genmatrix_bytes(SETS[name])
    elif op != "dec_onekey":
        ops += KECCAK_OPS * gen_a
    return nbytes, ops


def work(case):
    if case["op"] == "matvec":
        l, n = case["l"], case["n"]
        return {"bytes": n * (l * l * 512 + l * 256 + l * 512), "flops": n * l * l * 2 * 65536}
    pairs = _groups(case) if case["op"] == "dec_mixed" else [(case["set"], case["n"])]
    kind = {"dec_host": "dec", "dec_mixed": "dec"}.get(case["op"], case["op"])
    per = [(n, _instance_work(kind, name)) for name, n in pairs]
    return {"bytes": sum(n * w[0] for n, w in per), "flops": sum(n * w[1] for n, w in per)}


def exact(case, seed):
    """The matrix-vector product in 64 bits (a twisted FFT whose values stay
    far below 2^53, rounded); the KEM's outputs are bytes and have no such value."""
    if case["op"] != "matvec":
        return None
    st = prepare(case, seed)
    A = st["A"].transpose(1, 2) if case["transpose"] else st["A"]
    w = torch.exp(1j * math.pi * torch.arange(256, device="cuda", dtype=torch.float64) / 256)
    out = []
    for A_, s_ in zip(A.split(2048), st["s"].split(2048)):
        fa = torch.fft.fft(A_.to(torch.float64) * w)
        fs = torch.fft.fft(s_.to(torch.float64) * w)
        c = torch.fft.ifft((fa * fs[:, None]).sum(2)) * w.conj()
        out.append(c.real.round().to(torch.int64) & ((1 << case["eq"]) - 1))
    return torch.cat(out).to(torch.int16)
