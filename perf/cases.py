"""The calls whose time matters, as a user of shell_gpu.py makes them.

Every case is one call (the wire case two) of the library on device buffers, in
the shapes of the benchmark and the tests: RNS ciphertexts over six 45-bit or
up to twelve 50-bit primes with the 2^20 gadget, PIR queries modulo a 60-bit
prime with the 2^8 gadget, BFV over six main and seven auxiliary primes.  The
context and the keys are what a server creates once and keeps; prepare() makes
the ciphertexts of one request and the buffers of its result.

All results are residues, plaintext integers or packed bytes: whole numbers,
which have one right value, so there is no exact() in floating point.
"""
import ctypes
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "shell-encryption_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import shell_gpu as sg  # noqa: E402

# 1 mod 2^15 (rings up to n = 2^14) and 1 mod 2^16 (up to n = 2^15).
Q45 = [35184371138561, 35184370941953, 35184370352129, 35184370155521,
       35184369893377, 35184368877569]
Q50 = [1125899904679937, 1125899903827969, 1125899903500289, 1125899903107073,
       1125899902124033, 1125899901665281, 1125899899174913, 1125899896160257,
       1125899887312897, 1125899886395393, 1125899885740033, 1125899885412353]
Q60 = [1152921504606830593]
P45_AUX = [35184368320513, 35184368025601, 35184367828993, 35184367337473, 35184366911489,
           35184366551041, 35184366223361]
T = 65537
LOG_B = 20       # RNS gadgets
PIR_LOG_B = 8    # PIR gadget
VARIANCE = 8     # encryption error


def listed():
    return [
        # One ciphertext product of an interactive request: launches and
        # latency count, nothing fills the GPU.
        {"name": "mul_relin_one", "kind": "mul_relin", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 1},
        # The benchmark's batch: 1024 pairs, larger than L2 by far.
        {"name": "mul_relin_batch", "kind": "mul_relin", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 1024},
        # The deepest ring of the mixed and served workloads, an odd batch.
        {"name": "mul_relin_deep", "kind": "mul_relin", "log_n": 15, "limbs": 12, "bits": 50,
         "count": 21},
        # A group of the mixed workload in a small ring with few limbs.
        {"name": "mul_relin_small_ring", "kind": "mul_relin", "log_n": 12, "limbs": 2,
         "bits": 50, "count": 77},
        # Galois rotations of a batch (sums over slots, matrix products).
        {"name": "rotate_batch", "kind": "rotate", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 250, "step": 3},
        # Coefficient form to NTT form of a batch of polynomials.
        {"name": "ntt_forward", "kind": "ntt_forward", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 512},
        # And back, single-modulus ciphertexts over a 60-bit prime, ragged.
        {"name": "ntt_inverse_60", "kind": "ntt_inverse", "log_n": 12, "limbs": 1, "bits": 60,
         "count": 515},
        # Modulus switching of a batch of ciphertexts (two components each).
        {"name": "modreduce", "kind": "modreduce", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 128},
        # A PIR server's step: queries expanded and absorbed, 2^10 items.
        {"name": "pir", "kind": "pir", "log_n": 12, "levels": 10, "items": 1024, "count": 24},
        # Encryption of a batch with the randomness drawn on the device.
        {"name": "encrypt", "kind": "encrypt", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 200},
        # BFV products without relinearization.
        {"name": "bfv_mul", "kind": "bfv_mul", "log_n": 14, "limbs": 6, "bits": 45,
         "count": 96},
        # Results packed for the wire and requests unpacked.
        {"name": "wire", "kind": "wire", "log_n": 14, "limbs": 6, "bits": 45, "count": 256},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """Another case of the same ranges; counts spread over their logarithm and
    bounded so that no drawn case costs more than mul_relin_batch."""
    kind = rng.choice(["mul_relin", "mul_relin", "rotate", "ntt_forward", "ntt_inverse",
                       "modreduce", "pir", "encrypt", "bfv_mul", "wire"])
    if kind == "pir":
        levels = rng.randint(6, 10)
        return {"kind": kind, "log_n": 12, "levels": levels,
                "items": rng.randint((1 << levels) // 2 + 1, 1 << levels),
                "count": _log_uniform(rng, 1, 30 << (10 - levels))}
    if kind == "bfv_mul":
        return {"kind": kind, "log_n": 14, "limbs": 6, "bits": 45,
                "count": _log_uniform(rng, 1, 400)}
    if kind in ("ntt_forward", "ntt_inverse") and rng.random() < 0.3:
        log_n = rng.randint(11, 12)
        return {"kind": kind, "log_n": log_n, "limbs": 1, "bits": 60,
                "count": _log_uniform(rng, 1, 8192)}
    log_n = rng.randint(11, 15)
    bits = 50 if log_n == 15 else rng.choice([45, 50])
    limbs = rng.randint(2 if kind == "modreduce" else 1, 6 if bits == 45 else 12)
    case = {"kind": kind, "log_n": log_n, "limbs": limbs, "bits": bits}
    if kind in ("mul_relin", "rotate"):
        cost = (limbs * 3 * limbs) << log_n
        most = min(1024, (1024 * 6 * 18 << 14) // cost)
        if kind == "rotate":
            case["step"] = rng.randint(1, 8)
    else:
        most = min(4096, (512 * 6 << 14) // (limbs << log_n))
    case["count"] = _log_uniform(rng, 1, most)
    return case


def _primes(case):
    if case["kind"] == "pir":
        return Q60
    return {45: Q45, 50: Q50, 60: Q60}[case["bits"]][:case["limbs"]]


def _uniform(qs, shape, gen):
    """Uniform residues [..., len(qs), n], limb l below qs[l]."""
    out = torch.empty(shape, dtype=torch.int64, device="cuda")
    for l, q in enumerate(qs):
        out[..., l, :] = torch.randint(0, q, shape[:-2] + shape[-1:], dtype=torch.int64,
                                       device="cuda", generator=gen)
    return out


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


class _Handles:
    """The context and keys that a server of this case's shape keeps."""

    def __init__(self, case):
        kind, qs = case["kind"], _primes(case)
        log_n, n = case["log_n"], 1 << case["log_n"]
        self.ctx = sg.Context(log_n, qs, T, P45_AUX if kind == "bfv_mul" else ())
        gen = _generator(20240229)

        def key(log_b, power):
            k = sum(-(-q.bit_length() // log_b) for q in qs)
            rows = [_uniform(qs, (k, len(qs), n), gen).cpu().numpy() for _ in range(2)]
            return sg.Key(self.ctx, [log_b] * len(qs), power, *rows)

        if kind == "mul_relin":
            self.key = key(LOG_B, 1)
        elif kind == "rotate":
            self.key = key(LOG_B, pow(5, case["step"], 2 * n))
        elif kind == "pir":
            self.keys = [key(PIR_LOG_B, (n >> j) + 1) for j in range(case["levels"])]
            self.key_list = (ctypes.c_void_p * case["levels"])(*[k.h for k in self.keys])
            self.db = _uniform(qs, (case["items"], 1, n), gen)
        elif kind == "encrypt":
            self.secret = _uniform(qs, (len(qs), n), gen)
        elif kind == "modreduce":
            self.ql_inv = self.ctx.ql_inv(len(qs) - 1)


_kept = {}


def _handles(case):
    """One set of handles at a time: the requests of a server share them."""
    shape = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "count")))
    if shape not in _kept:
        _kept.clear()
        _kept[shape] = _Handles(case)
    return _kept[shape]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.h = case, _handles(case)
    kind, qs, count = case["kind"], _primes(case), case["count"]
    L, n = len(qs), 1 << case["log_n"]
    gen = _generator(seed)

    def empty(*shape):
        return torch.empty(shape, dtype=torch.int64, device="cuda")

    if kind == "mul_relin":
        s.a, s.b = (_uniform(qs, (count, 2, L, n), gen) for _ in range(2))
        s.out = empty(count, 2, L, n)
    elif kind == "rotate":
        s.ct = _uniform(qs, (count, 2, L, n), gen)
        s.out = empty(count, 2, L, n)
    elif kind in ("ntt_forward", "ntt_inverse"):
        s.polys = _uniform(qs, (count, L, n), gen)
    elif kind == "modreduce":
        s.ct = _uniform(qs, (count, 2, L, n), gen)
        s.out = empty(count, 2, L - 1, n)
    elif kind == "pir":
        s.ct = _uniform(qs, (count, 2, 1, n), gen)
        s.out = empty(count, 2, 1, n)
    elif kind == "encrypt":
        s.seeds = torch.randint(0, 256, (count, 32), dtype=torch.uint8, device="cuda",
                                generator=gen)
        s.m = _uniform(qs, (count, L, n), gen)
        s.out = empty(count, 2, L, n)
    elif kind == "bfv_mul":
        s.a, s.b = (_uniform(qs, (count, 2, L, n), gen) for _ in range(2))
        s.out = empty(count, 3, L, n)
    elif kind == "wire":
        s.ct = _uniform(qs, (count, 2, L, n), gen)
        s.back = empty(count, 2, L, n)
        per = sg.lib().shg_poly_serialized_bytes(s.h.ctx.h, L)
        s.packed = torch.empty(2 * count * per, dtype=torch.uint8, device="cuda")
    return s


def run(s):
    lib, ctx, case = sg.lib(), s.h.ctx.h, s.case
    kind, count = case["kind"], case["count"]
    if kind == "mul_relin":
        sg.check(lib.shg_bgv_mul_relin(ctx, s.h.key.h, s.out.data_ptr(), s.a.data_ptr(),
                                       s.b.data_ptr(), count, None))
        return s.out
    if kind == "rotate":
        sg.check(lib.shg_bgv_rotate(ctx, s.h.key.h, s.out.data_ptr(), s.ct.data_ptr(), count,
                                    None))
        return s.out
    if kind in ("ntt_forward", "ntt_inverse"):
        # In place: the next pass transforms what this one left.
        call = lib.shg_ntt_forward if kind == "ntt_forward" else lib.shg_ntt_inverse
        sg.check(call(ctx, s.polys.data_ptr(), count, case["limbs"], None))
        return s.polys
    if kind == "modreduce":
        ql = s.h.ql_inv.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))
        sg.check(lib.shg_poly_modreduce_lsb(ctx, s.out.data_ptr(), s.ct.data_ptr(), T, ql, 1,
                                            2 * count, case["limbs"], None))
        return s.out
    if kind == "pir":
        sg.check(lib.shg_pir_expand_absorb(ctx, s.h.key_list, case["levels"],
                                           s.h.db.data_ptr(), case["items"], s.out.data_ptr(),
                                           s.ct.data_ptr(), count, None))
        return s.out
    if kind == "encrypt":
        sg.check(lib.shg_bgv_encrypt(ctx, s.out.data_ptr(), s.h.secret.data_ptr(),
                                     s.m.data_ptr(), s.seeds.data_ptr(), case["limbs"], count,
                                     VARIANCE, None))
        return s.out
    if kind == "bfv_mul":
        sg.check(lib.shg_bfv_mul(ctx, s.out.data_ptr(), s.a.data_ptr(), s.b.data_ptr(), count,
                                 case["limbs"], None))
        return s.out
    sg.check(lib.shg_poly_serialize(ctx, s.packed.data_ptr(), s.ct.data_ptr(), 2 * count,
                                    case["limbs"], None))
    sg.check(lib.shg_poly_deserialize(ctx, s.back.data_ptr(), s.packed.data_ptr(), 2 * count,
                                      case["limbs"], None))
    return {"packed": s.packed, "back": s.back}


def work(case):
    """Bytes: each operand, key and database item read once, each result
    written once.  There is no floating-point work on this path."""
    kind, qs, count = case["kind"], _primes(case), case["count"]
    L, n = len(qs), 1 << case["log_n"]
    poly = L * n * 8
    if kind in ("mul_relin", "rotate"):
        dim = sum(-(-q.bit_length() // LOG_B) for q in qs)
        polys = (6 if kind == "mul_relin" else 4) * count + 2 * dim
    elif kind in ("ntt_forward", "ntt_inverse"):
        polys = 2 * count
    elif kind == "modreduce":
        polys = 2 * count * (1 + (L - 1) / L)
    elif kind == "pir":
        dim = -(-qs[0].bit_length() // PIR_LOG_B)
        polys = 4 * count + case["items"] + 2 * dim * case["levels"]
    elif kind == "encrypt":
        polys = 3 * count + 1
    elif kind == "bfv_mul":
        polys = 7 * count
    else:
        packed = sum(q.bit_length() for q in qs) / (64 * L)
        polys = 2 * count * (2 + 2 * packed)
    return {"bytes": polys * poly, "flops": 0}
