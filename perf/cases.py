"""Timing cases of the BFV evaluator: what programs built on it have it do.

Each case is one call sequence through the public classes (`BFVContext`,
`BFVScheme`, `MulPlan`) on ciphertexts that are real encryptions of uniform
slot vectors. A program makes its parameter sets and keys once and keeps them
(`session`); `prepare` makes the inputs of one pass from the seed.

The parameter sets are those of the request server's rings, the batched
multiply and transform benchmarks, the parameter sweep of the tests and the
reference's own two sets.
"""
import functools

import torch

import kunpbfv_b200 as kb

# name: (log2 N, ciphertext prime bits, special prime bits, plain modulus, key-switch digits)
RINGS = {
    "n4096": (12, [36, 36], [37], 65537, 2),
    "n8192": (13, [50, 50, 50], [52], 65537, 3),
    "n16384": (14, [60] * 7, [60], 65537, 1),
    "n16384_d7": (14, [60] * 7, [60], 65537, 7),
    "n32768": (15, [60] * 14, [60, 60], 65537, 3),
    "n65536": (16, [60] * 4, [60, 60], 786433, 2),
    "n65536_q32": (16, [60] * 32, [60], 786433, 1),
    # the reference's parameter sets, with the T base of its own key switch
    "ref14": (14, [35] * 4, [40] * 2, 23068673, 2),
    "ref15": (15, [55] * 15, [56], 786433, 15),
}
T_PRIMES = {"ref14": (4, 3, 2), "ref15": (4, 4, 15)}  # T primes, Ri blocks, Qj blocks
KEY_SEED = bytes(range(7, 39))


@functools.lru_cache(maxsize=3)
def session(ring, relin="hybrid"):
    """(context, secret key, scheme with its keys): what a program holds for its whole life."""
    if ring in T_PRIMES:
        ctx = kb.reference_context(RINGS[ring][0])
    else:
        log_n, q_bits, p_bits, t, dnum = RINGS[ring]
        ctx = kb.BFVContext.from_bits(log_n, q_bits, p_bits, t, dnum=dnum)
    sk = kb.SecretKey(ctx, KEY_SEED)
    scheme = kb.BFVScheme(ctx, KEY_SEED, relin=relin)
    scheme.addEncKey(sk)
    scheme.addMultKey_23(sk)
    return ctx, sk, scheme


def listed():
    return [
        # one small product: the first program that anybody writes, all launch latency
        {"name": "mul_n4096_1", "kind": "mul", "ring": "n4096", "count": 1, "plan": False},
        # a serving iteration of a middle ring: a few requests at once, one digit per prime
        {"name": "mul_n8192_5", "kind": "mul", "ring": "n8192", "count": 5, "plan": False},
        # a request loop with fixed buffers: one product per graph launch
        {"name": "mul_n16384_1_plan", "kind": "mul", "ring": "n16384", "count": 1, "plan": True},
        # throughput: the batched multiply at its benchmark size
        {"name": "mul_n16384_64", "kind": "mul", "ring": "n16384", "count": 64, "plan": False},
        # a circuit whose operands stand at four depths
        {"name": "levels_n32768_16", "kind": "levels", "ring": "n32768", "count": 16, "depths": 4},
        # the reference's own parameters and key switch, an odd small batch
        {"name": "klss_ref15_3", "kind": "klss", "ring": "ref15", "count": 3},
        # a rotation step over a batch (inner sums, matrix-vector products)
        {"name": "rotate_n16384_8", "kind": "rotate", "ring": "n16384_d7", "count": 8, "steps": 3},
        # the client's side: encode and encrypt, decrypt and decode
        {"name": "encrypt_n16384_64", "kind": "encrypt", "ring": "n16384", "count": 64},
        {"name": "decrypt_n16384_33", "kind": "decrypt", "ring": "n16384", "count": 33},
        # an affine layer without a key switch: (x + y) * w + b, then one level down
        {"name": "affine_n32768_7", "kind": "affine", "ring": "n32768", "count": 7},
        # bare transforms: the whole prime chain over 64 polynomials, and an odd number of rows
        {"name": "ntt_fwd_n65536_2048", "kind": "ntt", "ring": "n65536_q32", "rows": 2048, "forward": True},
        {"name": "ntt_inv_n16384_333", "kind": "ntt", "ring": "n16384", "rows": 333, "forward": False},
    ]


# the largest batch that a drawn case takes from a ring, by kind
MOST = {
    "mul": {"n4096": 128, "n8192": 64, "n16384": 64, "n16384_d7": 24, "n32768": 9, "n65536": 8},
    "levels": {"n8192": 32, "n16384_d7": 16, "n32768": 14},
    "klss": {"ref14": 64, "ref15": 8},
    "rotate": {"n8192": 64, "n16384": 64, "n16384_d7": 24, "n32768": 12},
    "encrypt": {"n4096": 128, "n8192": 128, "n16384": 64, "n32768": 16},
    "decrypt": {"n4096": 128, "n8192": 128, "n16384": 64, "n32768": 16},
    "affine": {"n8192": 128, "n16384": 48, "n32768": 12},
    "ntt": {"n4096": 2047, "n8192": 2047, "n16384": 2047, "n32768": 2047, "n65536_q32": 2047},
}


def draw(rng):
    """One more case of these kinds: any ring of the kind, sizes spread over their logarithm."""
    kind = rng.choice(("mul", "mul", "mul", "levels", "klss", "rotate", "encrypt", "decrypt", "affine", "ntt"))
    ring = rng.choice(sorted(MOST[kind]))
    size = int(round(MOST[kind][ring] ** rng.random()))
    if kind == "ntt":
        return {"kind": kind, "ring": ring, "rows": size, "forward": rng.random() < 0.5}
    case = {"kind": kind, "ring": ring, "count": size}
    if kind == "mul":
        case["plan"] = size <= 4 and rng.random() < 0.5
    if kind == "levels":
        case["count"] = max(2, size)
        case["depths"] = rng.randint(2, len(RINGS[ring][1]) if ring == "n8192" else 4)
    if kind == "rotate":
        case["steps"] = rng.randint(1, 64)
    return case


def slots(ctx, count, gen):
    return torch.randint(0, ctx.plain_modulus, (count, ctx.N), dtype=torch.int64, device="cuda", generator=gen)


def encryption(ctx, scheme, count, gen, enc_id):
    return scheme.encryptMsg(kb.Plaintext(ctx, ctx.encode(slots(ctx, count, gen))), enc_id=enc_id)


def prepare(case, seed):
    kind, ring = case["kind"], case["ring"]
    ctx, sk, scheme = session(ring, "klss" if kind == "klss" else "hybrid")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    enc_id = seed << 12  # each seed's encryptions have randomness of their own
    state = {"kind": kind, "ctx": ctx, "sk": sk, "scheme": scheme}
    if kind == "ntt":
        # uniform residues, row r over prime r mod q_count: evaluations and coefficients look alike
        rows = torch.empty(case["rows"], ctx.N, dtype=torch.int64, device="cuda")
        for i, q in enumerate(ctx.q):
            part = rows[i::ctx.q_count]
            if part.numel():
                part.copy_(torch.randint(0, q, part.shape, dtype=torch.int64, device="cuda", generator=gen))
        state.update(rows=rows, forward=case["forward"])
        return state
    count = case["count"]
    if kind == "encrypt":
        state.update(slots=slots(ctx, count, gen), enc_id=enc_id)
        return state
    if kind == "levels":
        top, state["pairs"] = ctx.q_count, []
        for j in range(count):
            ab = encryption(ctx, scheme, 2, gen, enc_id + 2 * j)
            ab = scheme.mod_switch_to(ab, top - j % case["depths"])
            both = ab.cipher_device.view(2, -1)
            state["pairs"].append((kb.Ciphertext(ab.ctx, both[0]), kb.Ciphertext(ab.ctx, both[1])))
        return state
    state["a"] = encryption(ctx, scheme, count, gen, enc_id)
    if kind in ("mul", "klss", "affine"):
        state["b"] = encryption(ctx, scheme, count, gen, enc_id + count)
    if kind == "mul" and case["plan"]:
        state["plan"] = scheme.mult_relin_plan(state["a"], state["b"], kb.Ciphertext(ctx, count=count))
    if kind == "rotate":
        state["g"] = scheme.galois_element(case["steps"])
        scheme.addGaloisKey(sk, state["g"])
    if kind == "affine":
        state["w"] = ctx.encode_ntt(ctx.encode(slots(ctx, count, gen)))
        state["bias"] = kb.Plaintext(ctx, ctx.encode(slots(ctx, count, gen)))
    return state


def run(state):
    kind, ctx, scheme = state["kind"], state["ctx"], state["scheme"]
    if kind == "ntt":  # in place
        (ctx.ntt_fwd if state["forward"] else ctx.ntt_inv)(state["rows"], 0, ctx.q_count)
        return state["rows"]
    if kind == "encrypt":
        return scheme.encryptMsg(kb.Plaintext(ctx, ctx.encode(state["slots"])), enc_id=state["enc_id"]).cipher_device
    if kind == "decrypt":
        return ctx.decode(scheme.decryptMsg(state["sk"], state["a"]).mx_device)
    if kind == "rotate":
        return scheme.apply_galois(state["a"], state["g"]).cipher_device
    if kind == "levels":
        return [out.cipher_device for out in scheme.mult_relin_levels(state["pairs"])]
    if kind == "affine":
        out = scheme.add(state["a"], state["b"])
        scheme.multConstAndEqual(out, state["w"])
        scheme.addConstAndEqual(out, state["bias"])
        return scheme.mod_switch(out).cipher_device
    if "plan" in state:
        return state["plan"].launch().cipher_device
    return scheme.mult_relin(state["a"], state["b"]).cipher_device


def transform_products(log_n):
    """modular products of one limb's transform"""
    return log_n * 2 ** (log_n - 1)


def multiply_products(log_n, q, p, dnum, key_switch):
    """modular products of one ciphertext multiply: transforms, base extensions, tensor, key product"""
    r, n = q + 1, 2 ** log_n
    limbs = 4 * q + 4 * r + 3 * (q + r)
    coeff = 4 * q * r + 3 * r * (q + 1) + 3 * r * q + 4 * (q + r)
    if key_switch == "hybrid":
        limbs += dnum * (q + p) + 2 * p + 2 * q
        coeff += q * (q + p) + 2 * dnum * (q + p)
    else:
        t, ri, qj = key_switch
        limbs += qj * t + 2 * ri * t + 2 * q
        coeff += q * t + 2 * ri * qj * t + 2 * (q + p) * t
    return limbs * transform_products(log_n) + coeff * n


def work(case):
    """Bytes of the inputs, keys and outputs, each once; every modular product counted as two operations."""
    log_n, q_bits, p_bits, _, dnum = RINGS[case["ring"]]
    q, p, n = len(q_bits), len(p_bits), 2 ** log_n
    poly, ct, count = 8 * n, 16 * q * n, case.get("count", 0)
    key = 16 * dnum * (q + p) * n
    kind = case["kind"]
    if kind == "ntt":
        rows = case["rows"]
        return {"bytes": rows * 2 * poly + 16 * n * min(rows, q), "flops": 2 * rows * transform_products(log_n)}
    if kind == "levels":
        live = [q - j % case["depths"] for j in range(count)]
        alpha = -(-q // dnum)
        ops = sum(multiply_products(log_n, k, p, -(-k // alpha), "hybrid") for k in live)
        return {"bytes": sum(48 * k * n for k in live) + key, "flops": 2 * ops}
    if kind == "klss":
        t, ri, qj = T_PRIMES[case["ring"]]
        ops = count * multiply_products(log_n, q, p, dnum, (t, ri, qj))
        return {"bytes": count * 3 * ct + 2 * qj * ri * t * poly, "flops": 2 * ops}
    if kind == "mul":
        return {"bytes": count * 3 * ct + key, "flops": 2 * count * multiply_products(log_n, q, p, dnum, "hybrid")}
    if kind == "rotate":
        limbs = q + dnum * (q + p) + 2 * p + 2 * q
        ops = limbs * transform_products(log_n) + (q * (q + p) + 2 * dnum * (q + p)) * n
        return {"bytes": count * 2 * ct + key, "flops": 2 * count * ops}
    if kind == "encrypt":
        ops = (1 + 4 * q) * transform_products(log_n) + 2 * q * n
        return {"bytes": count * (poly + ct) + ct, "flops": 2 * count * ops}
    if kind == "decrypt":
        ops = (1 + q) * transform_products(log_n) + 2 * q * n
        return {"bytes": count * (poly + ct) + poly * q, "flops": 2 * count * ops}
    ops = (q + 2 + 2 * (q - 1)) * transform_products(log_n) + (2 * q + q + 2 * (q - 1)) * n
    return {"bytes": count * (2 * ct + poly * q + poly + 16 * (q - 1) * n), "flops": 2 * count * ops}


def exact(case, seed):
    """Every output is an array of residues: whole numbers, equal or wrong."""
    return None
