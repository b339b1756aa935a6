"""The work a user of this library has it do, case by case, through its public entry points.

A case is a dict of plain values; `op` says which call it makes, the rest its sizes:

  log_n    ring degree 2^log_n
  chain    Q primes of the modulus chain: one of 60 bits and chain - 1 of `bits` bits
  limbs    Q primes the input still has (limbs < chain: a ciphertext deeper in the chain)
  special  special primes of 60 bits (digits of the key decomposition hold that many limbs)

Contexts, keys, Galois tables and pre-encoded matrices are made once per parameter set and kept, as a server keeps
them; every state gets inputs of its own. The parameter sets are those of the tests (rings of 2^12 to 2^16), of the
benchmark (2^14 with 8 limbs of 50 bits; 2^16 with 24 limbs and 8 special primes) and of the bootstrapping example.
"""
import collections
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "phantom-fhe_b200"))
import pyPhantom as ph  # noqa: E402
from pyPhantom import linalg  # noqa: E402
from pyPhantom._native import LIB, check  # noqa: E402

SCALE = 2.0 ** 40
KEY_SEED = 20  # keys, secrets and matrices belong to the parameter set, not to the inputs


# ---- the cases ----------------------------------------------------------------------------------------------------
def listed():
    return [
        # the transforms alone: the benchmark's small configuration, one polynomial forward and one back
        dict(name="ntt_n14_l8", op="ntt", log_n=14, limbs=8, bits=50),
        # one product near the end of a short chain in the smallest ring: launches and host calls count
        dict(name="product_n12_l3", op="product", log_n=12, chain=3, limbs=3, special=1, bits=40),
        # one product of the headline configuration, as an interactive circuit issues them
        dict(name="product_n16_l24", op="product", log_n=16, chain=24, limbs=24, special=8, bits=40),
        # one slot rotation two levels down a medium chain, with a digit that is not full
        dict(name="rotate_n13_l7", op="rotate", log_n=13, chain=9, limbs=7, special=3, bits=40, step=1),
        # the baby steps of a linear transform: eight rotations of one ciphertext from one decomposition
        dict(name="hoist_n15_l12_s8", op="hoist", log_n=15, chain=12, limbs=12, special=4, bits=40, steps=8),
        # a batch of independent products in a mid-sized ring (products of attention scores, squarings of a batch)
        dict(name="products_n14_l8_b32", op="products", log_n=14, chain=8, limbs=8, special=2, bits=40, batch=32),
        # the headline benchmark's call: a batch of relinearisations that share one key
        dict(name="relin_n16_l24_b16", op="relin", log_n=16, chain=24, limbs=24, special=8, bits=40, batch=16),
        # a client's round trip: host values encoded, encrypted, decrypted, decoded back to host values
        dict(name="client_n15_l9", op="client", log_n=15, chain=9, limbs=9, special=2, bits=40),
        # an activation function: a polynomial of one ciphertext (the degree of bootstrapping's cosine halved)
        dict(name="poly_n15_d31", op="poly", log_n=15, chain=14, limbs=14, special=3, bits=40, degree=31),
        # a layer's matrix product with the diagonals kept on the host, the reference's driver
        dict(name="matvec_n14_d256", op="matvec", log_n=14, chain=6, limbs=6, special=2, bits=40, d_pad=256, baby=16),
        # a layer's matrix product with the diagonals resident in device memory
        dict(name="matvec_hbm_n16_d1024", op="matvec_hbm", log_n=16, chain=16, limbs=16, special=8, bits=40, d_pad=1024, baby=32),
        # bootstrapping at full size on the benchmark's chain; the result is decrypted, as its precision is what counts
        dict(name="bootstrap_n16", op="bootstrap", log_n=16, user=8, special=8),
    ]


def _log_int(rng, lo, hi):
    """an integer of [lo, hi], spread evenly over the logarithm"""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    """one more case of the ranges that the listed ones stand for"""
    op = rng.choice(["ntt", "product", "rotate", "hoist", "products", "relin", "client", "poly", "matvec", "matvec_hbm", "bootstrap"])
    if op == "ntt":
        return dict(op=op, log_n=rng.randint(12, 17), limbs=_log_int(rng, 1, 32), bits=rng.choice([30, 36, 40, 45, 50, 58]))
    if op in ("product", "rotate", "hoist", "products", "relin"):
        chain = _log_int(rng, 2, 24)
        c = dict(op=op, log_n=rng.randint(12, 17 if op in ("product", "rotate") else 16), chain=chain,
                 limbs=rng.choice([chain, rng.randint(2, chain)]), special=_log_int(rng, 1, min(8, chain)), bits=rng.choice([30, 36, 40, 40, 50]))
        if op == "rotate":
            c["step"] = rng.choice([1, -1, 2, 5, 16, 100, -64])
        if op == "hoist":
            c["steps"] = _log_int(rng, 2, 16)
        if op in ("products", "relin"):
            # up to 64 sets in small rings, at most the headline's 16 x 24 limbs of 2^16 in all
            c["batch"] = _log_int(rng, 2, max(2, min(64, (16 * 24 << 16) // (c["limbs"] << c["log_n"]))))
        return c
    if op == "client":
        chain = _log_int(rng, 2, 24)
        return dict(op=op, log_n=rng.randint(12, 16), chain=chain, limbs=rng.choice([chain, rng.randint(2, chain)]), special=rng.randint(1, 3), bits=40)
    if op == "poly":
        degree = _log_int(rng, 3, 63)
        chain = _poly_levels(degree) + rng.randint(2, 5)
        return dict(op=op, log_n=rng.randint(12, 16), chain=chain, limbs=chain, special=rng.randint(2, 4), bits=40, degree=degree)
    if op == "matvec":
        chain = rng.randint(3, 8)
        d_pad = 1 << rng.randint(4, 8)
        return dict(op=op, log_n=rng.randint(12, 15), chain=chain, limbs=rng.randint(2, chain), special=rng.randint(1, 3), bits=40, d_pad=d_pad,
                    baby=1 << rng.randint(1, d_pad.bit_length() - 2))
    if op == "matvec_hbm":
        chain = rng.randint(4, 16)
        d_pad = 1 << rng.randint(5, 9)
        return dict(op=op, log_n=rng.randint(12, 16), chain=chain, limbs=chain, special=rng.randint(2, 6), bits=40, d_pad=d_pad,
                    baby=1 << ((d_pad.bit_length() - 1) // 2))
    return dict(op=op, log_n=rng.randint(12, 15), user=rng.randint(2, 8), special=rng.randint(3, 7))


def _poly_levels(degree):
    m = math.ceil(math.sqrt(degree + 1))
    return m + (degree + m) // m - 2


# ---- what a parameter set keeps -------------------------------------------------------------------------------------
_KITS = collections.OrderedDict()
_MOST_KITS = 3


def _kit(case, make):
    """the parameter set's context, keys and plans: made on first use, the least recently used ones dropped"""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "batch", "limbs")) + [("limbs", case.get("limbs") if case["op"] in ("ntt", "matvec_hbm") else 0)])
    if key in _KITS:
        _KITS.move_to_end(key)
    else:
        while len(_KITS) >= _MOST_KITS:
            _KITS.popitem(last=False)
        _KITS[key] = make(case)
    return _KITS[key]


def _context(log_n, bit_sizes, special, steps=()):
    N = 1 << log_n
    parms = ph.params(ph.scheme_type.ckks)
    parms.set_poly_modulus_degree(N)
    parms.set_coeff_modulus(ph.create_coeff_modulus(N, bit_sizes))
    parms.set_special_modulus_size(special)
    parms.set_galois_elts(sorted({ph.get_elt_from_step(s, N) for s in steps} | {2 * N - 1}))
    return ph.context(parms)


def _bits(case):
    return [60] + [case["bits"]] * (case["chain"] - 1) + [60] * case["special"]


def _residues(ctx, gen, *lead, primes):
    """[*lead][len(primes)][N] residues, uniform below each prime, as ciphertext and key limbs are"""
    out = torch.empty(*lead, len(primes), ctx.N, dtype=torch.int64, device="cuda")
    for i, q in enumerate(primes):
        out[..., i, :] = torch.randint(0, int(q), (*lead, ctx.N), generator=gen, device="cuda", dtype=torch.int64)
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ciphertext(ctx, data, limbs):
    ct = ph.ciphertext()
    ct._chain_index, ct._size, ct._N, ct._limbs, ct._scale = ctx.size_Q - limbs + 1, data.shape[0], ctx.N, limbs, SCALE
    ct.data = data
    return ct


def _switching_key(ctx, gen):
    """a key of uniform limbs: the arithmetic does not depend on whose secret it encrypts"""
    k = ph.relin_key()
    for _ in range(ctx.beta(ctx.size_Q)):
        ct = ph.ciphertext()
        ct._chain_index, ct._size, ct._N, ct._limbs = 0, 2, ctx.N, ctx.size_QP
        ct.data = _residues(ctx, gen, 2, primes=ctx.primes)
        k.public_keys.append(ct)
    return k


def _hoist_steps(case):
    return list(range(1, case["steps"] + 1))


def _make_switching(case):
    steps = [case["step"]] if case["op"] == "rotate" else _hoist_steps(case) if case["op"] == "hoist" else []
    ctx, gen = _context(case["log_n"], _bits(case), case["special"], steps), _gen(KEY_SEED)
    if not steps:
        return dict(ctx=ctx, rlk=_switching_key(ctx, gen))
    return dict(ctx=ctx, steps=steps, glk=ph.galois_key.from_keys([_switching_key(ctx, gen) for _ in ctx.galois_elts]))


def _make_ntt(case):
    return dict(ctx=_context(case["log_n"], [case["bits"]] * case["limbs"] + [60], 1))


def _make_client(case):
    ctx = _context(case["log_n"], _bits(case), case["special"])
    return dict(ctx=ctx, sk=ph.secret_key(ctx, seed=KEY_SEED), enc=ph.ckks_encoder(ctx))


def _encryptor(kit, seed):
    """the parameter set's secret with an encryption randomness of its own"""
    sk = ph.secret_key(seed=int(seed))
    sk.data = kit["sk"].data
    return sk


def _encrypted(kit, values, limbs, seed):
    ctx = kit["ctx"]
    pt = kit["enc"].encode_double_vector(ctx, values, SCALE, chain_index=ctx.size_Q - limbs + 1)
    return _encryptor(kit, seed).encrypt_symmetric(ctx, pt)


def _make_poly(case):
    ctx = _context(case["log_n"], _bits(case), case["special"])
    sk = ph.secret_key(ctx, seed=KEY_SEED)
    # coefficients of an activation's size: values in [-1, 1] stay of order one
    coeffs = np.random.default_rng(KEY_SEED).uniform(-1.0, 1.0, case["degree"] + 1) / (1.0 + np.arange(case["degree"] + 1))
    return dict(ctx=ctx, sk=sk, enc=ph.ckks_encoder(ctx), rlk=sk.gen_relinkey(ctx), coeffs=coeffs)


def _random_diagonals(case, ctx):
    """pre-encoded diagonals: the signed coefficients of an encoded weight matrix look like rounded Gaussians"""
    rng = np.random.default_rng(KEY_SEED)
    block = rng.normal(0.0, 2.0 ** 30, ctx.N + case["d_pad"]).astype(np.int64)  # a window of it for each diagonal
    scps = [ph.single_chain_plaintext(block[d: d + ctx.N], SCALE) for d in range(case["d_pad"])]
    return ph.bsgs_diagonals(scps, case["d_pad"], case["baby"], case["d_pad"] // case["baby"])


def _make_matvec(case):
    ctx = _context(case["log_n"], _bits(case), case["special"], ph.bsgs_required_steps(case["baby"]))
    gen = _gen(KEY_SEED)
    return dict(ctx=ctx, glk=ph.galois_key.from_keys([_switching_key(ctx, gen) for _ in ctx.galois_elts]), diags=_random_diagonals(case, ctx))


def _make_matvec_hbm(case):
    M, G = case["baby"], case["d_pad"] // case["baby"]
    steps = list(range(1, M)) + [g * M for g in range(1, G)]
    ctx = _context(case["log_n"], _bits(case), case["special"], steps)
    sk = ph.secret_key(ctx, seed=KEY_SEED)
    glk = sk.create_galois_keys(ctx)
    mat = linalg.resident_bsgs(ctx, glk, _random_diagonals(case, ctx), ctx.size_Q - case["limbs"] + 1)
    return dict(ctx=ctx, sk=sk, enc=ph.ckks_encoder(ctx), mat=mat)


def _make_bootstrap(case):
    log_n, N = case["log_n"], 1 << case["log_n"]
    parms = ph.params(ph.scheme_type.ckks)
    parms.set_poly_modulus_degree(N)
    parms.set_special_modulus_size(case["special"])
    parms.set_coeff_modulus(ph.create_coeff_modulus(N, [58] + [40] * case["user"] + [58] * 12 + [29] * 3 + [58] * case["special"]))
    parms.set_galois_elts(ph.bootstrap_required_galois_elts(log_n))
    ctx = ph.context(parms)
    sk = ph.secret_key(ctx, seed=KEY_SEED)
    sk.generate_sparse(ctx, 192)
    enc = ph.ckks_encoder(ctx)
    bk = ph.create_bootstrap_key(ctx, enc, sk, sparse_hamming_weight=192, eval_mod_levels=9, user_scale=SCALE)
    kit = dict(ctx=ctx, sk=sk, enc=enc, bk=bk)
    for _ in range(2):  # a server's warm-up: the second call captures the graph that later ones replay
        ph.bootstrap(ctx, enc, _depleted(kit, KEY_SEED), bk, SCALE)
    return kit


def _depleted(kit, seed):
    """a ciphertext of slots in [-0.4, 0.4] with two limbs left"""
    return _encrypted(kit, np.random.default_rng(seed).uniform(-0.4, 0.4, kit["ctx"].N // 2), 2, seed)


_MAKERS = dict(ntt=_make_ntt, client=_make_client, poly=_make_poly, matvec=_make_matvec, matvec_hbm=_make_matvec_hbm, bootstrap=_make_bootstrap)


# ---- inputs, one pass, its work and how exact it is ------------------------------------------------------------------
def prepare(case, seed):
    op = case["op"]
    kit = _kit(case, _MAKERS.get(op, _make_switching))
    ctx, gen = kit["ctx"], _gen(seed)
    s = dict(kit, op=op, case=case)
    if op == "ntt":
        s["fwd"] = _residues(ctx, gen, primes=ctx.primes[: case["limbs"]])
        s["inv"] = _residues(ctx, gen, primes=ctx.primes[: case["limbs"]])
        return s
    l = case.get("limbs", 0)
    if op in ("product", "rotate", "hoist", "matvec"):
        s["a"] = _ciphertext(ctx, _residues(ctx, gen, 2, primes=ctx.primes[:l]), l)
        if op == "product":
            s["b"] = _ciphertext(ctx, _residues(ctx, gen, 2, primes=ctx.primes[:l]), l)
    elif op == "products":
        s["a"], s["b"] = (_residues(ctx, gen, case["batch"], 2, primes=ctx.primes[:l]) for _ in range(2))
    elif op == "relin":
        s["data"] = _residues(ctx, gen, case["batch"], 3, primes=ctx.primes[:l])
    elif op == "client":
        rng = np.random.default_rng(seed)
        s["values"] = rng.uniform(-1.0, 1.0, ctx.N // 2) + 1j * rng.uniform(-1.0, 1.0, ctx.N // 2)
        s["sk"] = _encryptor(kit, seed)
    elif op in ("poly", "matvec_hbm"):
        z = np.random.default_rng(seed).uniform(-1.0, 1.0, ctx.N // 2)
        s["x"] = _encrypted(kit, z, l, seed)
    elif op == "bootstrap":
        s["x"] = _depleted(kit, seed)
    return s


def _read(s, ct):
    """the slots of a result, on the device"""
    return s["enc"].decode_complex_tensor(s["ctx"], s["sk"].decrypt(s["ctx"], ct))


def run(s):
    op, ctx, case = s["op"], s["ctx"], s["case"]
    if op == "ntt":
        stream = torch.cuda.current_stream().cuda_stream
        check(LIB.b2_ntt_forward(ctx._h, s["fwd"].data_ptr(), case["limbs"], 0, stream))
        check(LIB.b2_ntt_inverse(ctx._h, s["inv"].data_ptr(), case["limbs"], 0, stream))
        return s["fwd"], s["inv"]
    if op == "product":
        return ph.rescale_to_next(ctx, ph.multiply_and_relin(ctx, s["a"], s["b"], s["rlk"])).data
    if op == "rotate":
        return ph.rotate(ctx, s["a"], case["step"], s["glk"]).data
    if op == "hoist":
        return [c.data for c in ph.hoist_rotations(ctx, s["a"], s["glk"], s["steps"])]
    if op == "products":
        return ph.multiply_relin_rescale_batch(ctx, s["a"], s["b"], s["rlk"])
    if op == "relin":
        return ph.relinearize_batch(ctx, s["data"], s["rlk"])
    if op == "client":
        l = case["limbs"]
        pt = s["enc"].encode_complex_vector(ctx, s["values"], SCALE, chain_index=ctx.size_Q - l + 1)
        return s["enc"].decode_complex_vector(ctx, s["sk"].decrypt(ctx, s["sk"].encrypt_symmetric(ctx, pt)))
    if op == "poly":
        return _read(s, ph.eval_polynomial(ctx, s["enc"], s["rlk"], s["x"], s["coeffs"]))
    if op == "matvec":
        return ph.bsgs_matmul_preencoded(ctx, s["glk"], s["a"], s["diags"]).data
    if op == "matvec_hbm":
        return _read(s, s["mat"].apply(s["x"]))
    return _read(s, ph.bootstrap(ctx, s["enc"], s["x"], s["bk"], SCALE))


def work(case):
    """bytes: inputs, keys and plaintexts read once, results written once. flops: an NTT butterfly counts three
    operations (a modular product, a sum, a difference), a modular multiply-add two; the transforms and conversions of
    a key switch are those of the hybrid method."""
    op, N = case["op"], 1 << case["log_n"]
    limb, ntt = 8.0 * N, 1.5 * N * case["log_n"]
    if op == "ntt":
        return {"bytes": 4 * case["limbs"] * limb, "flops": 2 * case["limbs"] * ntt}
    a = case["special"]

    def key(l):
        return 2 * -(-l // a) * (l + a)

    def switch(l, outs=1):
        """transforms, conversions and inner products, the decomposition shared by `outs` results"""
        beta = -(-l // a)
        up = (l + beta * (l + a) - l) * ntt + 2 * N * beta * l * min(a, l)
        down = (2 * a + 2 * l) * ntt + 4 * N * a * l + 4 * N * beta * (l + a)
        return up + outs * down

    if op == "bootstrap":
        l = case["user"] + 8  # half way down
        steps = len(ph.bootstrap_required_galois_elts(case["log_n"]))
        return {"bytes": (steps * key(l) + 4 * l) * limb + 16.0 * N, "flops": (steps + 40) * switch(l)}
    l = case["limbs"]
    if op == "product":
        return {"bytes": (4 * l + 2 * (l - 1) + key(l)) * limb, "flops": switch(l) + 2 * l * ntt + 8 * N * l}
    if op == "rotate":
        return {"bytes": (4 * l + key(l)) * limb, "flops": switch(l)}
    if op == "hoist":
        k = case["steps"]
        return {"bytes": (2 * l + k * (2 * l + key(l))) * limb, "flops": switch(l, k)}
    if op == "products":
        b = case["batch"]
        return {"bytes": (b * (4 * l + 2 * (l - 1)) + key(l)) * limb, "flops": b * (switch(l) + 2 * l * ntt + 8 * N * l)}
    if op == "relin":
        b = case["batch"]
        return {"bytes": (5 * b * l + key(l)) * limb, "flops": b * switch(l)}
    if op == "client":
        return {"bytes": 16.0 * N + l * limb, "flops": 4 * l * ntt + 10.0 * N * case["log_n"]}
    if op == "poly":
        muls = 2 * math.ceil(math.sqrt(case["degree"] + 1))
        return {"bytes": (2 * l + key(l)) * limb + 8.0 * N, "flops": muls * switch(l - _poly_levels(case["degree"]) // 2)}
    M, G = case["baby"], case["d_pad"] // case["baby"]
    if op == "matvec":
        keys = len(ph.bsgs_required_steps(M))
        return {"bytes": (case["d_pad"] + 4 * l + keys * key(l)) * limb, "flops": (M + G - 2) * switch(l) + case["d_pad"] * l * (ntt + 4 * N)}
    return {"bytes": (case["d_pad"] * l + 2 * l + (M + G - 2) * key(l)) * limb + 8.0 * N,
            "flops": switch(l, M - 1) + (G - 1) * switch(l) + 4.0 * N * case["d_pad"] * l}


def tolerance(case):
    """Limbs are whole numbers with one right value each. Decrypted slots carry the scheme's own rounding (units of
    2^-40 times the ring's expansion; bootstrapping's approximation of the modular reduction, about 2^-20)."""
    return {"client": {"rel": 1e-8}, "poly": {"rel": 1e-6}, "matvec_hbm": {"rel": 1e-6}, "bootstrap": {"rel": 1e-5}}.get(case["op"], "exact")
