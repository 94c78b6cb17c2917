"""Performance cases of the framework: what a CKKS program has it do, through the public entry points.

Three parameter sets, all of them the repository's own (``cerium_b200/params.py``):

  rot64   N = 2^16, 35 primes of 50 bits, 5 extension primes of 60 bits, digits of up to 5 limbs
          (``config_hrot``; at level L a ciphertext has L limbs and ceil(L / 5) digits)
  mul64   first prime 60 bits, 23 of 50 bits, one 60-bit extension prime, one digit per limb
          (``config_hmult``)
  ref32   the reference's chain of 64 primes of 28 bits, 13 of them extension primes, digits of up to 13
          limbs (``config_ref28``)

64-bit sets use the exact base conversion and rounding, the 32-bit set the reference's lazy conversion and
floor division: the semantics each is used with.  Ciphertexts, keys and plaintexts are uniform residues,
which is what encrypted data looks like to the kernels.  Contexts and key-switching plans are kept for the
life of the process, as a program keeps them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cerium_b200 import _capi, bootstrap, params, runtime
from cerium_b200.bsgs import BsgsMultiplyAccumulate

LOGN = 16
N = 1 << LOGN
DIGIT = {"rot64": 5, "mul64": 1, "ref32": 13}    # limbs of a full digit
TOP = {"rot64": 35, "mul64": 24, "ref32": 51}    # limbs of a fresh ciphertext
EXT = {"rot64": 5, "mul64": 1, "ref32": 13}      # extension primes


def listed():
    return [
        # addition of two ciphertexts near the end of a computation: the smallest call, two short launches
        {"name": "add_rot64_L6", "op": "add", "set": "rot64", "L": 6},
        # plaintext product and rescale at a middle level with an odd limb count: the step of every linear layer
        {"name": "mul_plain_rescale_rot64_L13", "op": "mul_plain", "set": "rot64", "L": 13},
        # inverse transform of one low-level polynomial (decoding, level management): few blocks, latency
        {"name": "ntt_inverse_rot64_7", "op": "ntt", "set": "rot64", "count": 7, "inverse": True},
        # batched forward transforms, 8 polynomials of 48 limbs: the stand-alone transform throughput
        {"name": "ntt_forward_rot64_384", "op": "ntt", "set": "rot64", "count": 384, "inverse": False},
        # rotation of a fresh ciphertext: the headline operation
        {"name": "hrot_rot64_L35", "op": "hrot", "set": "rot64", "L": 35},
        # the same two thirds down the chain, with ragged digits (4 + 4 + 4 of at most 5 limbs)
        {"name": "hrot_rot64_L12", "op": "hrot", "set": "rot64", "L": 12},
        # multiplication, relinearisation and rescale with one digit per limb
        {"name": "hmult_mul64_L24", "op": "hmult", "set": "mul64", "L": 24, "rescale": 2},
        # the 28-bit chain of the reference's programs: rotation of a fresh ciphertext, wide digits
        {"name": "hrot_ref32_L51", "op": "hrot", "set": "ref32", "L": 51},
        # ... and a multiplication in the middle of such a program, rescaled by a division of its own
        {"name": "hmult_ref32_L27", "op": "hmult", "set": "ref32", "L": 27, "rescale": 1},
        # one 64-diagonal linear transform (matrix-vector product, CoeffToSlot stage)
        {"name": "bsgs_rot64_L35_8x8", "op": "bsgs", "set": "rot64", "L": 35, "baby": 8, "giant": 8},
        # a whole bootstrap: ModRaise, 3 + 3 linear stages, degree-63 polynomial, double angles
        {"name": "bootstrap_rot64_34_8x8", "op": "bootstrap", "set": "rot64", "top": 34, "stages": 3, "baby": 8, "giant": 8},
        # the client's side: a message of 2^15 slots encoded and encrypted, and the result decrypted and decoded
        {"name": "client_ref32_L17", "op": "client", "set": "ref32", "L": 17, "bits": 40},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["add", "mul_plain", "ntt", "ntt", "hrot", "hrot", "hrot", "hmult", "hmult", "bsgs", "bootstrap", "client"])
    if op == "add":
        s = rng.choice(["rot64", "ref32"])
        return {"op": op, "set": s, "L": _log_uniform(rng, 2, TOP[s])}
    if op == "mul_plain":
        s = rng.choice(["rot64", "ref32"])
        return {"op": op, "set": s, "L": _log_uniform(rng, 3, TOP[s])}
    if op == "ntt":
        return {"op": op, "set": rng.choice(["rot64", "rot64", "ref32"]), "count": _log_uniform(rng, 1, 384), "inverse": rng.random() < 0.5}
    if op == "hrot":
        s = rng.choice(["rot64", "rot64", "ref32"])
        return {"op": op, "set": s, "L": rng.randint(3, TOP[s])}
    if op == "hmult":
        s = rng.choice(["mul64", "rot64", "ref32"])
        return {"op": op, "set": s, "L": rng.randint(4, TOP[s]), "rescale": rng.choice([0, 1, 2])}
    if op == "bsgs":
        return {"op": op, "set": "rot64", "L": rng.randint(6, 35), "baby": rng.randint(3, 8), "giant": rng.randint(2, 8)}
    if op == "bootstrap":
        stages = rng.choice([2, 3])
        return {"op": op, "set": "rot64", "top": rng.randint(2 * stages + 11, 34), "stages": stages,
                "baby": rng.choice([4, 8]), "giant": rng.choice([4, 8])}
    return {"op": "client", "set": "ref32", "L": rng.randint(3, 17), "bits": rng.randint(28, 44)}


# ---------------------------------------------------------------------------------------------------------
# what a program keeps: contexts, plans, and the keys of a bootstrap
# ---------------------------------------------------------------------------------------------------------

_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _set(name):
    """(parameters, library context) of a set; the 32-bit one is the runtime surface's context."""
    def make():
        if name == "rot64":
            prm = params.config_hrot()
        elif name == "mul64":
            prm = params.config_hmult()
        else:
            prm = params.config_ref28(L=TOP[name], K=EXT[name], dnum=4)
            rt = runtime.Context(N // 2, prm.moduli, device=torch.cuda.current_device())
            return prm, rt.handle, rt
        return prm, _capi.Context(_capi.load(), prm.moduli, prm.word_bits, device=torch.cuda.current_device()), None
    return _keep(("set", name), make)


def _dnum(name, L):
    return -(-L // DIGIT[name])


def _plan(name, L):
    prm, ctx, _ = _set(name)
    modes = (_capi.BCONV_LAZY, _capi.ROUND_FLOOR) if prm.word_bits == 32 else (_capi.BCONV_EXACT, _capi.ROUND_HALF)
    return _keep(("plan", name, L), lambda: _capi.KeySwitch(ctx, prm.q_idx[:L], prm.p_idx, _dnum(name, L), *modes))


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _limbs(prm, idx, lead, gen):
    """[lead..., len(idx), N] uniform residues, one word each."""
    q = torch.tensor([prm.moduli[p] for p in idx], dtype=torch.int64, device="cuda").view(-1, 1)
    x = torch.randint(0, 1 << 62, tuple(lead) + (len(idx), N), dtype=torch.int64, device="cuda", generator=gen)
    x.remainder_(q)
    return x if prm.word_bits == 64 else x.to(torch.int32)


def _new(prm, *shape):
    return torch.empty(shape + (N,), dtype=torch.int64 if prm.word_bits == 64 else torch.int32, device="cuda")


def _bootstrap(case):
    """The evaluator of one bootstrap shape with its keys and diagonals on the device; one shape is kept at a time."""
    shape = bootstrap.BootstrapShape(top=case["top"], stages=case["stages"], baby=case["baby"], giant=case["giant"])
    key = ("bootstrap", case["top"], case["stages"], case["baby"], case["giant"])
    if key not in _kept:
        for k in [k for k in _kept if k[0] == "bootstrap"]:
            del _kept[k]
        torch.cuda.empty_cache()
        prm, ctx, _ = _set("rot64")
        lib = _capi.load()
        gen = torch.Generator(device="cuda").manual_seed(0xB007)
        # bootstrap() takes the last rung of the chain for the prime that ModRaise divides away
        material = bootstrap.BootstrapMaterial(prm.moduli, prm.q_idx, prm.p_idx, prm.dnum, shape,
                                               lambda tag, lead, idx: _limbs(prm, list(idx), lead, gen),
                                               lambda step: lib.galois_elt_from_step(step, LOGN))
        ev = bootstrap.GpuEvaluator(torch, _capi, ctx, material, _capi.BCONV_EXACT, _capi.ROUND_HALF)
        ev.stream = _stream()
        bootstrap.bootstrap(ev, shape, [_limbs(prm, prm.q_idx[:2], (), gen) for _ in range(2)])  # makes every level's keys
        _kept[key] = ev
    return shape, _kept[key]


# ---------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    op, name = case["op"], case["set"]
    prm, ctx, rt = _set(name)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = {"case": case, "prm": prm, "ctx": ctx}
    if op == "bootstrap":
        s["shape"], s["ev"] = _bootstrap(case)
        s["ct"] = [_limbs(prm, prm.q_idx[:2], (), gen) for _ in range(2)]
        return s
    if op == "client":
        rng = np.random.default_rng(seed)
        sk = np.zeros(N, dtype=np.int64)
        sk[rng.choice(N, 192, replace=False)] = rng.choice([-1, 1], 192)
        ectx = runtime.CKKSEncryptorContext(rt, sk)
        s["enc"] = runtime.CKKSEncryptor(ectx, prng_seed=[seed, 1])
        s["message"] = rng.uniform(-1, 1, N // 2) + 1j * rng.uniform(-1, 1, N // 2)
        return s
    if op == "ntt":
        # polynomials at a fresh ciphertext's level, back to back; the last one is cut short
        s["idx"] = [prm.q_idx[i % TOP[name]] for i in range(case["count"])]
        s["x"] = _limbs(prm, s["idx"], (), gen)
        s["out"] = torch.empty_like(s["x"])
        return s
    L = case["L"]
    q = s["q"] = prm.q_idx[:L]
    s["a"] = _limbs(prm, q, (2,), gen)
    if op == "add":
        s["b"] = _limbs(prm, q, (2,), gen)
        s["out"] = _new(prm, 2, L)
        return s
    if op == "mul_plain":
        s["pt"] = _limbs(prm, q, (), gen)
        s["prod"], s["scratch"], s["out"] = _new(prm, 2, L), _new(prm, 2), _new(prm, 2, L - 1)
        return s
    ks = s["ks"] = _plan(name, L)
    key = lambda: _limbs(prm, q + prm.p_idx, (_dnum(name, L), 2), gen)  # noqa: E731
    lib = _capi.load()
    if op == "hrot":
        s["key"] = key()
        s["elt"] = lib.galois_elt_from_step(1 + seed % (N // 2 - 1), LOGN)
        s["out"] = _new(prm, 2, L)
    elif op == "hmult":
        s["key"] = key()
        s["b"] = _limbs(prm, q, (2,), gen)
        s["out"] = _new(prm, 2, L - (1 if case["rescale"] else 0))
    else:  # bsgs: diagonals in bootstrapping's use, the rescale in the same division
        g, ng = case["baby"], case["giant"]
        s["op"] = BsgsMultiplyAccumulate(ctx, ks, g, ng, lambda shape: torch.empty(tuple(shape), dtype=torch.int64, device="cuda"),
                                         lambda t: t.data_ptr(), rescale_levels=1)
        s["pts"] = [[_limbs(prm, q, (), gen) for _ in range(g)] for _ in range(ng)]
        s["baby_keys"] = [key() for _ in range(g - 1)]
        s["giant_keys"] = [key() for _ in range(ng - 1)]
        s["baby_elts"] = [lib.galois_elt_from_step(i, LOGN) for i in range(1, g)]
        s["giant_elts"] = [lib.galois_elt_from_step(g * j, LOGN) for j in range(1, ng)]
        s["out"] = _new(prm, 2, L - 1)
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    op = case["op"]
    if op == "bootstrap":
        s["ev"].stream = _stream()
        ct = bootstrap.bootstrap(s["ev"], s["shape"], s["ct"])
        return [ct.c0[:ct.level], ct.c1[:ct.level]]
    if op == "client":
        ct = s["enc"].encode_and_encrypt(s["message"], 2.0 ** case["bits"], list(range(case["L"])))
        return {"c0": ct.c0.view(np.int32), "c1": ct.c1.view(np.int32), "message": s["enc"].decrypt_and_decode(ct, 2.0 ** case["bits"])}
    out, st = s["out"], _stream()
    if op == "ntt":
        (ctx.ntt_inverse if case["inverse"] else ctx.ntt_forward)(out.data_ptr(), s["x"].data_ptr(), s["idx"], stream=st)
        return out
    a = s["a"]
    if op == "add":
        for p in range(2):
            ctx.ewise(_capi.EW_ADD, out[p].data_ptr(), a[p].data_ptr(), s["q"], b=s["b"][p].data_ptr(), stream=st)
    elif op == "mul_plain":
        prod = s["prod"]
        for p in range(2):
            ctx.ewise(_capi.EW_MUL, prod[p].data_ptr(), a[p].data_ptr(), s["q"], b=s["pt"].data_ptr(), stream=st)
        ctx.rescale(out.data_ptr(), prod.data_ptr(), s["q"], 2, s["scratch"].data_ptr(),
                    _capi.ROUND_HALF if ctx.word_bits == 64 else _capi.ROUND_FLOOR, st)
    elif op == "hrot":
        s["ks"].hrot(out[0].data_ptr(), out[1].data_ptr(), a[0].data_ptr(), a[1].data_ptr(), s["key"].data_ptr(), s["elt"], st)
    elif op == "hmult":
        b = s["b"]
        s["ks"].hmult(out[0].data_ptr(), out[1].data_ptr(), a[0].data_ptr(), a[1].data_ptr(), b[0].data_ptr(), b[1].data_ptr(),
                      s["key"].data_ptr(), case["rescale"], st)
    else:
        s["op"].run(out, a, s["pts"], s["baby_keys"], s["giant_keys"], s["baby_elts"], s["giant_elts"], st)
    return out


# ---------------------------------------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------------------------------------

_BUTTERFLIES = N // 2 * LOGN  # of one limb transform


def _keyswitch(name, L, raises=1, keys=1, downs=1):
    """(limbs of key read, modular products) of `keys` key switches sharing `raises` ModUps and `downs` ModDowns."""
    d, K = _dnum(name, L), EXT[name]
    raised = d * (L + K) - L
    butterflies = raises * (L + raised) + downs * (2 * K + 2 * L)
    conv = 0 if DIGIT[name] == 1 else raised * -(-L // d)
    products = butterflies * _BUTTERFLIES + N * (raises * conv + keys * 2 * d * (L + K) + downs * 2 * L * (K + 1))
    return keys * 2 * d * (L + K), products


def work(case):
    """bytes: every input read once, every output written once.  flops: two per modular product (the product and
    the sum or difference it goes into); they run on the integer and double-precision pipes."""
    op, name = case["op"], case["set"]
    limb = N * (4 if name == "ref32" else 8)
    if op == "ntt":
        return {"bytes": 2 * case["count"] * limb, "flops": 2 * case["count"] * _BUTTERFLIES}
    if op == "client":
        # 2^15 complex slots in and out, the ciphertext out; coefficients and key are taken modulo every prime
        L = case["L"]
        return {"bytes": 2 * (N // 2) * 16 + 2 * L * limb, "flops": 2 * (3 * L * _BUTTERFLIES + 4 * L * N)}
    if op == "bootstrap":
        return _bootstrap_work(case, limb)
    L = case["L"]
    if op == "add":
        return {"bytes": 6 * L * limb, "flops": 2 * L * N}
    if op == "mul_plain":
        return {"bytes": (3 * L + 2 * (L - 1)) * limb, "flops": 2 * (2 * L * N + 2 * L * _BUTTERFLIES + 2 * L * N)}
    if op == "hrot":
        keys, products = _keyswitch(name, L)
        return {"bytes": (4 * L + keys) * limb, "flops": 2 * products}
    if op == "hmult":
        keys, products = _keyswitch(name, L)
        out = L - (1 if case["rescale"] else 0)
        return {"bytes": (4 * L + keys + 2 * out) * limb, "flops": 2 * (products + 4 * L * N)}
    g, ng = case["baby"], case["giant"]
    keys, products = _keyswitch(name, L, raises=ng, keys=g - 1 + ng - 1, downs=g)
    return {"bytes": (2 * L + keys + g * ng * L + 2 * (L - 1)) * limb, "flops": 2 * (products + 2 * g * ng * L * N)}


def _bootstrap_work(case, limb):
    top, g, ng, stages = case["top"], case["baby"], case["giant"], case["stages"]
    limbs, products = 4 + 2 * (top + 1 + EXT["rot64"]), 0   # the input and the key of ModRaise
    level = top

    def switch(level, **how):
        nonlocal products
        keys, prod = _keyswitch("rot64", level, **how)
        products += prod
        return keys

    def linear(level):
        nonlocal limbs, products
        limbs += switch(level, raises=1 + ng, keys=g - 1 + ng, downs=g) + (g * ng - 1) * level
        products += 2 * (g * ng - 1) * level * N

    for _ in range(stages):
        linear(level)
        level -= 1
    limbs += switch(level)                                   # conjugation
    # both parts: T_2 .. T_8 over three levels, then a level for the coefficients, three for the giant
    # steps (T_16 and T_32 on the way) and one for each double angle; a level's key is read once
    for depth, mults in enumerate([1, 2, 4, 1, 5, 2, 1, 1, 1]):
        keys = 0
        for _ in range(2 * mults):
            keys = switch(level - depth)
        limbs += keys
    limbs += 8 * 7 * (level - 3)
    level -= 9
    for _ in range(stages):
        linear(level)
        level -= 1
    return {"bytes": (limbs + 2 * level) * limb, "flops": 2 * products}


def tolerance(case):
    if case["op"] == "client":
        # the ciphertext is exact; the slots pass through one double-precision FFT of 2^16 points each way
        return {"rel": 1e-12, "max": 1e-10}
    return "exact"
