"""The work a CKKS program has this framework do, case by case.

Every case goes through the public entry points: ``CkksEngine`` methods, the
mixed-batch executor and the bootstrapping object.  The kinds:

``hmult``      multiply -> relinearise -> rescale of a batch in one call
``steps``      the same as the three separate calls
``rotate``     one rotation of a batch with a key the program holds
``matvec``     matrix-vector product by diagonals: hoisted rotations, a
               plaintext product each, their sum and one rescale
``mixed``      a batch of ciphertexts at their own levels, each with its own
               operation (a multiplication or a rotation)
``to_ntt``     coefficient -> NTT domain
``from_ntt``   NTT -> coefficient domain
``client``     encode + encrypt messages, and decrypt + decode received ones
``bootstrap``  full-slot bootstrapping of exhausted ciphertexts

Ciphertext and key residues are uniform modulo their primes, which is how
real ciphertexts and keys look to the evaluator; ``client`` and ``bootstrap``
use real messages, keys and encryptions.  The engine (its tables) and the
bootstrapping object (its keys and diagonals) are what a program builds once
and keeps, so they are shared by the states of one configuration.
"""

from __future__ import annotations

import math
from functools import lru_cache

import torch

from fhelium_b200.batch import MixedItemsExecutor, sample_mixed_workload
from fhelium_b200.bootstrap import FullSlotBootstrap
from fhelium_b200.config import CkksConfig, Preset
from fhelium_b200.engine import CkksEngine
from fhelium_b200.values import (Ciphertext, EncryptionDraws, Plaintext, RelinearizationKey, RotationKey)

MIXED_STEPS = (1, -2, 16, -128, 1024, 4096)  # the rotation steps a mixed program holds keys for


def listed():
    return [
        # the smallest call a program makes: one ciphertext of the smallest ring, where latency counts
        dict(name="hmult_n14_b1", kind="hmult", preset="slots8192_scale40_levels7_int64", level=2, batch=1),
        # an odd small batch in the middle ring, part of the way down the chain
        dict(name="hmult_n15_b5", kind="hmult", preset="slots16384_scale40_levels16_int64", level=3, batch=5),
        # the throughput workload: a full batch at the top of the deepest 40-bit chain of N = 2^16
        dict(name="hmult_n16_b32", kind="hmult", preset="slots32768_scale40_levels34_int64", level=0, batch=32),
        # the same on the 50-bit chain that high-precision programs and bootstrapping use
        dict(name="hmult_n16_s50_b6", kind="hmult", preset="slots32768_scale50_levels27_int64", level=1, batch=6),
        # the 32-bit residue family, written as three separate calls
        dict(name="steps_n15_i32_b9", kind="steps", preset="slots16384_scale25_levels29_int32", level=4, batch=9),
        # one rotation of one ciphertext in the middle of a computation
        dict(name="rotate_n16_b1", kind="rotate", preset="slots32768_scale40_levels34_int64", level=20, batch=1, step=5),
        # a matrix-vector product of eight diagonals
        dict(name="matvec_n16_d8_b3", kind="matvec", preset="slots32768_scale40_levels34_int64", level=6, batch=3,
             diagonals=8),
        # a server's queue: ciphertexts of many programs, each at its own level
        dict(name="mixed_n16_48", kind="mixed", preset="slots32768_scale40_levels34_int64", count=48, workload=7),
        # domain changes on their own, 64-bit forward and 32-bit inverse
        dict(name="to_ntt_n16_b12", kind="to_ntt", preset="slots32768_scale40_levels34_int64", level=0, batch=12),
        dict(name="from_ntt_n16_i32_b48", kind="from_ntt", preset="slots32768_scale25_levels24_int32", level=0,
             batch=48),
        # the client: a few messages encrypted, a few results decrypted
        dict(name="client_n15_b3", kind="client", preset="slots16384_scale40_levels16_int64", level=0, batch=3),
        # a whole pipeline: bootstrapping a pair of ciphertexts
        dict(name="bootstrap_n16_b2", kind="bootstrap", log_n=16, batch=2),
    ]


# the presets a drawn case takes: every ring and both word sizes, with the batch that stays below the largest case
DRAW_PRESETS = {
    "slots8192_scale30_levels9_int64": 64, "slots8192_scale40_levels7_int64": 64,
    "slots8192_scale50_levels5_int64": 64, "slots8192_scale25_levels14_int32": 64,
    "slots16384_scale30_levels21_int64": 32, "slots16384_scale40_levels16_int64": 32,
    "slots16384_scale50_levels12_int64": 32, "slots16384_scale25_levels29_int32": 32,
    "slots32768_scale30_levels45_int64": 16, "slots32768_scale40_levels34_int64": 24,
    "slots32768_scale50_levels27_int64": 16, "slots32768_scale25_levels24_int32": 32,
    "slots65536_scale40_levels72_int64": 3, "slots65536_scale25_levels14_int32": 16,
}


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.99)))))))


def draw(rng):
    kind = rng.choice(["hmult", "hmult", "hmult", "steps", "rotate", "rotate", "matvec", "matvec", "mixed", "to_ntt",
                       "from_ntt", "client", "bootstrap"])
    if kind == "bootstrap":
        return dict(kind=kind, log_n=rng.choice([12, 13, 14]), batch=rng.randint(1, 6))
    names = list(DRAW_PRESETS)
    if kind in ("mixed", "client"):
        names = [p for p in names if not p.startswith("slots65536")]
    preset = rng.choice(names)
    most = DRAW_PRESETS[preset]
    if kind == "mixed":
        return dict(kind=kind, preset=preset, count=rng.randint(6, 40), workload=rng.randint(0, 1 << 20))
    levels = CkksConfig.parse(Preset[preset]).num_scale_primes
    case = dict(kind=kind, preset=preset, level=rng.randint(0, levels - 1))
    if kind == "matvec":
        case.update(diagonals=rng.randint(2, 12), batch=_log_uniform(rng, 1, max(1, most // 8)))
    elif kind == "client":
        case.update(batch=_log_uniform(rng, 1, 9))
    elif kind in ("to_ntt", "from_ntt"):
        case.update(batch=_log_uniform(rng, 1, 2 * most))
    else:
        case.update(batch=_log_uniform(rng, 1, most))
    if kind == "rotate":
        case.update(step=rng.choice([-1, 1]) * rng.randint(1, 4000))
    return case


# ---------------------------------------------------------------------------
# what the program keeps
# ---------------------------------------------------------------------------
def _config(case):
    if case["kind"] == "bootstrap":
        if case["log_n"] == 16:
            return CkksConfig.parse(Preset.slots32768_scale50_levels27_int64, base_prime_bits=50)
        # the small rings of the tests: the same chain shape, below the security budget
        return CkksConfig(logN=case["log_n"], scale_bits=50, base_prime_bits=50, num_scale_primes=27, num_p_primes=4,
                          enforce_security_budget=False)
    return CkksConfig.parse(Preset[case["preset"]])


@lru_cache(maxsize=2)
def _engine(preset):
    return CkksEngine(CkksConfig.parse(Preset[preset]), rng_seed=1)


@lru_cache(maxsize=1)
def _bootstrap(log_n):
    eng = CkksEngine(_config(dict(kind="bootstrap", log_n=log_n)), galois_generator=5, rng_seed=3)
    boot = FullSlotBootstrap(eng)
    boot.generate_keys()
    boot.precompute()
    return eng, boot


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _uniform(eng, g, prefix, rows, lazy=False):
    """[*prefix, len(rows), N] residues uniform in [0, q), or [0, 2q) for the lazy NTT-domain state."""
    out = torch.empty((*prefix, len(rows), eng.n), dtype=eng.dtype, device=eng.device)
    for j, pid in enumerate(rows):
        q = eng.moduli[pid] * (2 if lazy else 1)
        out[..., j, :] = torch.randint(0, q, (*prefix, eng.n), generator=g, device=eng.device, dtype=torch.int64)
    return out


def _ciphertext(eng, g, batch, level, ntt):
    data = _uniform(eng, g, (2, batch), range(level, eng.num_q), lazy=ntt)
    state = ("ntt", "montgomery") if ntt else ("coefficient", "standard")
    return Ciphertext(data, level, eng.config.default_scale, *state)


def _key_data(eng, g):
    return _uniform(eng, g, (eng.key_digit_count, 2), range(eng.num_q + eng.num_p))


def _rotation_key(eng, g, step):
    return RotationKey(_key_data(eng, g), step, eng.galois_element_for_step(step))


def _message(eng, g, batch):
    re = torch.rand((batch, eng.num_slots), generator=g, device=eng.device, dtype=torch.float64) * 2 - 1
    im = torch.rand((batch, eng.num_slots), generator=g, device=eng.device, dtype=torch.float64) * 2 - 1
    return torch.complex(re, im)


def _draws(eng, g, batch):
    """The encryption's random values, from the seed like every other input."""
    shape = (batch, eng.n)

    def gaussian():
        x = torch.randn(shape, generator=g, device=eng.device, dtype=torch.float64) * eng.config.sigma
        return torch.round(x).to(torch.int64)

    v = torch.randint(-1, 2, shape, generator=g, device=eng.device, dtype=torch.int64)
    return EncryptionDraws(v, gaussian(), gaussian(),
                           torch.rand(shape, generator=g, device=eng.device, dtype=torch.float64))


def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    if kind == "bootstrap":
        eng, boot = _bootstrap(case["log_n"])
        msg, draws = _message(eng, g, case["batch"]), _draws(eng, g, case["batch"])
        ct = eng.encrypt_message(msg, level=eng.public_level_count - 1, draws=draws)
        return dict(kind=kind, boot=boot, ct=ct)
    eng = _engine(case["preset"])
    s = dict(kind=kind, eng=eng)
    if kind in ("hmult", "steps"):
        s["a"] = _ciphertext(eng, g, case["batch"], case["level"], True)
        s["b"] = _ciphertext(eng, g, case["batch"], case["level"], True)
        s["key"] = RelinearizationKey(_key_data(eng, g))
    elif kind == "rotate":
        s["ct"] = _ciphertext(eng, g, case["batch"], case["level"], False)
        s["key"] = _rotation_key(eng, g, case["step"])
    elif kind == "matvec":
        s["ct"] = _ciphertext(eng, g, case["batch"], case["level"], False)
        s["steps"] = list(range(case["diagonals"]))
        for step in s["steps"][1:]:
            eng.set_rotation_key(_rotation_key(eng, g, step))
        s["keys"] = [eng.rotation_key(step) for step in s["steps"][1:]]
        rows = range(case["level"], eng.num_q)
        s["diagonals"] = [Plaintext(None, case["level"], eng.config.default_scale, _uniform(eng, g, (), rows),
                                    representation="rns", polynomial_domain="ntt", modulus_basis="Q",
                                    residue_representation="montgomery", prime_ids=tuple(rows)) for _ in s["steps"]]
    elif kind == "mixed":
        levels, ops = sample_mixed_workload(eng.num_q, case["count"], seed=case["workload"])
        ops = [op if op.kind != "rotate_by_step" else type(op)(op.kind, op.index, op.partner,
                                                               MIXED_STEPS[op.step % len(MIXED_STEPS)]) for op in ops]
        cts = [Ciphertext(_uniform(eng, g, (2,), range(lv, eng.num_q)), lv, eng.config.default_scale)
               for lv in levels]
        eng.set_relinearization_key(RelinearizationKey(_key_data(eng, g)))
        for step in sorted({op.step for op in ops if op.kind == "rotate_by_step"}):
            eng.set_rotation_key(_rotation_key(eng, g, step))
        # the executor is the plan a program builds once for its batch and runs again
        s["executor"] = MixedItemsExecutor(eng, cts, ops, max_scratch_bytes=4 << 30)
    elif kind in ("to_ntt", "from_ntt"):
        s["ct"] = _ciphertext(eng, g, case["batch"], case["level"], kind == "from_ntt")
    elif kind == "client":
        s["message"] = _message(eng, g, case["batch"])
        s["draws"] = _draws(eng, g, case["batch"])
        s["level"] = case["level"]
        received = _message(eng, g, case["batch"])
        s["received"] = eng.encrypt_message(received, level=case["level"], draws=_draws(eng, g, case["batch"]))
    return s


def run(state):
    kind = state["kind"]
    if kind == "bootstrap":
        return state["boot"](state["ct"]).data
    eng = state["eng"]
    if kind == "hmult":
        return eng.multiply_relinearize_rescale(state["a"], state["b"], state["key"]).data
    if kind == "steps":
        product = eng.relinearize(eng.multiply(state["a"], state["b"]), state["key"])
        return eng.rescale_to_next_level(product).data
    if kind == "rotate":
        return eng.rotate_with_key(state["ct"], state["key"]).data
    if kind == "matvec":
        ct = state["ct"]
        rotated = [ct] + eng.rotate_many_with_keys(ct, state["keys"])
        total = None
        for r, diagonal in zip(rotated, state["diagonals"]):
            term = eng.multiply_plaintext(eng.coefficient_domain_to_ntt_domain(r), diagonal)
            total = term if total is None else eng.add(total, term)
        return eng.rescale_to_next_level(eng.ntt_domain_to_coefficient_domain(total)).data
    if kind == "mixed":
        state["executor"].run()
        return [ct.data for ct in state["executor"].results()]
    if kind == "to_ntt":
        return eng.coefficient_domain_to_ntt_domain(state["ct"]).data
    if kind == "from_ntt":
        return eng.ntt_domain_to_coefficient_domain(state["ct"]).data
    sent = eng.encrypt_message(state["message"], level=state["level"], draws=state["draws"])
    return {"sent": sent.data, "received": eng.decrypt_message(state["received"])}


def exact(case, seed):
    """Residues are whole numbers, equal or wrong, so only the client's
    decrypted slots have a value in 64 bits: the messages themselves."""
    if case["kind"] != "client":
        return None
    eng, g = _engine(case["preset"]), _generator(seed)
    _message(eng, g, case["batch"]), _draws(eng, g, case["batch"])  # the sent messages come first
    return {"sent": None, "received": _message(eng, g, case["batch"]).cpu()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _chain(case):
    cfg = _config(case)
    q, p = cfg.num_q_primes, cfg.num_p_primes
    return cfg.N, cfg.logN, q, p, 8 if cfg.buffer_bit_length == 62 else 4


def _ntt(n, log_n):
    return 2 * (n // 2) * log_n  # one modular product and one addition pair per butterfly


def _key_switch(n, log_n, q, p, level, relin):
    """Operations of one key switch at a level: ModUp's extension, the digits'
    forward transforms, the key products, the inverse transforms, ModDown."""
    l = q - level
    digits = sum(1 for s in range(0, q - 1, p) if min(s + p, q - 1) > level) + 1
    transforms = digits * (l + p) - (l if relin else 0)
    return (transforms * _ntt(n, log_n) + 2 * (l + p) * _ntt(n, log_n) + 2 * n * l * (l + p - 1)
            + 4 * n * digits * (l + p) + 4 * n * l * (p + 1)), digits


def work(case):
    n, log_n, q, p, w = _chain(case)
    kind = case["kind"]
    if kind == "bootstrap":
        # the transforms' diagonals and baby steps' keys once, 16 + 7 products of ciphertext pairs and the rotations
        b, steps, products = case["batch"], 60, 15 + 7
        per, digits = _key_switch(n, log_n, q, p, 8, True)
        keys = (steps + 2) * 2 * digits * (q + p) * n * w
        return {"bytes": keys + 2 * b * n * w * (1 + q - 18), "flops": b * per * (steps + 2 * products)}
    if kind == "mixed":
        levels, ops = sample_mixed_workload(q, case["count"], seed=case["workload"])
        nbytes, flops, keys = 0, 0, set()
        for op in ops:
            lv, mult = levels[op.index], op.kind != "rotate_by_step"
            l = q - lv
            per, _ = _key_switch(n, log_n, q, p, lv, mult)
            flops += per + (2 * 4 * n * l + 5 * l * _ntt(n, log_n) if mult else 0)
            nbytes += 2 * l * n * w * (2 if mult else 1) + 2 * (l - mult) * n * w
            keys.add("mult" if mult else MIXED_STEPS[op.step % len(MIXED_STEPS)])
        return {"bytes": nbytes + len(keys) * 2 * (-(-(q - 1) // p) + 1) * (q + p) * n * w, "flops": flops}
    level, b = case["level"], case["batch"]
    l = q - level
    ct = 2 * b * l * n * w
    if kind in ("to_ntt", "from_ntt"):
        return {"bytes": 2 * ct, "flops": 2 * b * l * _ntt(n, log_n)}
    if kind == "client":
        transforms = 4 * l + 2 * l + (2 * l + l)
        return {"bytes": 2 * ct + 2 * b * n * 8 + 5 * l * n * w, "flops": b * (transforms * _ntt(n, log_n) + 12 * n * log_n)}
    per, digits = _key_switch(n, log_n, q, p, level, kind in ("hmult", "steps"))
    key = 2 * digits * (l + p) * n * w
    if kind == "matvec":
        d = case["diagonals"]
        one, _ = _key_switch(n, log_n, q, p, level, False)
        hoisted = 2 * (l + p) * _ntt(n, log_n) + 4 * n * digits * (l + p) + 4 * n * l * (p + 1)
        flops = b * (one + (d - 2) * hoisted + 2 * (d + 1) * l * _ntt(n, log_n) + 4 * d * n * l)
        return {"bytes": 2 * ct + (d - 1) * key + d * l * n * w, "flops": flops}
    if kind == "rotate":
        return {"bytes": 2 * ct + key, "flops": b * per}
    return {"bytes": 2 * ct + 2 * b * (l - 1) * n * w + key,
            "flops": b * (per + 2 * 4 * n * l + l * _ntt(n, log_n))}
