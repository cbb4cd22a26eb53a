"""The work that users of this engine have it do, as measurable cases.

Every case is one pass through the engine's public entry points on inputs that
already lie on the GPU:

* ``gates``      cufhe_gate_batch: a batch of independent gates on Ctxt<lvl1>
                 (level 1), Ctxt<lvl0> (level 0) or Ctxt<lvl0> through lvl2
                 (level 2), one gate id for all or a mix, with either form of
                 the bootstrapping key (KeyBundle or plain) and either
                 precision form (FP64 FFNT, exact INT8)
* ``circuit``    cufhe_circuit_run: ripple-carry adders, dependent gates in
                 narrow waves, replayed from the circuit's CUDA graph
* ``keyswitch``  cufhe_identity_keyswitch: lvl1 -> lvl0 key switching alone
* ``lut``        cufhe_lut_eval: 8-bit lookup tables as CMUX trees

The keys are real keys of one fixed secret key, generated once per process and
uploaded when a case needs another set than the one on the device.  Circuit
bootstrapping is not a case of its own: its private key-switching keys are 5 GB
of host data, and 86 % of its time is the lvl0 -> lvl2 rotation that the level 2
gates run; the lookup tables it feeds are a case.

Outputs are Torus32 words modulo 2^32, compared bit for bit.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cufhepp_b200 import circuits, client, engine, params as P

# gates of the mixed batches: the headline benchmark's mix
MIX = [P.NAND, P.AND, P.OR, P.XOR, P.XNOR, P.MUX]
KEY_SEED = 20


def _gates(name, count, level=1, mix="mixed", key="kb", form="fp64"):
    return {"name": name, "kind": "gates", "count": count, "level": level, "mix": mix,
            "key": key, "form": form}


def listed():
    return [
        # one gate, the latency that an interactive program sees
        _gates("nand1", 1, mix="nand"),
        # a few Mux gates in the BR -> IKS order: one step of a small datapath
        _gates("mux16_lvl0", 16, level=0, mix="mux"),
        # an ordinary ragged batch, less than one resident wave of lanes
        _gates("mixed333", 333),
        # the 1000 random NAND pairs of the benchmark, plain bootstrapping key
        _gates("nand1000_plain", 1000, mix="nand", key="plain"),
        # the headline batch: 4096 gates over NAND/AND/OR/XOR/XNOR/MUX
        _gates("mixed4096", 4096),
        # a large odd batch in the BR -> IKS order
        _gates("mixed9001_lvl0", 9001, level=0),
        # the exact integer form, for callers that need bit-exact ciphertexts
        _gates("int8_mixed1000", 1000, form="int8"),
        # one gate through lvl2 (64-bit torus, larger message space)
        _gates("lvl02_nand1", 1, level=2, mix="nand"),
        # a ragged batch through lvl2
        _gates("lvl02_mixed700", 700, level=2),
        # dependent gates: 16 adders of 16 bits, 33 waves of 32 to 64 lanes
        {"name": "adders16x16", "kind": "circuit", "adders": 16, "width": 16},
        # key switching of a batch of ciphertexts
        {"name": "keyswitch4096", "kind": "keyswitch", "count": 4096},
        # 128 tables of 8 bits over circuit-bootstrapped bits (the benchmark's step)
        {"name": "lut128", "kind": "lut", "tables": 128},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["gates"] * 8 + ["circuit", "keyswitch", "lut"])
    if kind == "keyswitch":
        return {"kind": kind, "count": _log_int(rng, 1, 8192)}
    if kind == "lut":
        return {"kind": kind, "tables": _log_int(rng, 1, 256)}
    if kind == "circuit":
        return {"kind": kind, "adders": _log_int(rng, 1, 48), "width": rng.randint(4, 24)}
    what = rng.choice(["lvl1"] * 4 + ["lvl0"] * 2 + ["int8", "lvl02"])
    c = _gates("", 1, level={"lvl0": 0, "lvl02": 2}.get(what, 1),
               mix=rng.choice(["nand", "mixed", "mixed", "mux"]),
               key=rng.choice(["kb", "kb", "plain"]), form="int8" if what == "int8" else "fp64")
    del c["name"]
    c["count"] = _log_int(rng, 1, {"int8": 1000, "lvl02": 900}.get(what, 3000))
    return c


# ------------------------------------------------------------------ keys ----
_keys: dict = {}
_on_device = {"lvl1": None, "lvl02": None}


def _key(what, make):
    if what not in _keys:
        _keys[what] = make()
    return _keys[what]


def _secret():
    return _key("sk", lambda: client.SecretKey.generate(KEY_SEED))


def _load_keys(level, key):
    """The case's key set on the device (as a program's start-up does)."""
    sk = _secret()
    if level == 2:
        ek = _key(("lvl02", key), lambda: client.EvalKey02.generate(sk, keybundle=key == "kb"))
        if _on_device["lvl02"] != key:
            engine.initialize_lvl02(ek)
            _on_device["lvl02"] = key
    else:
        ek = _key(("lvl1", key), lambda: client.EvalKey.generate(sk, keybundle=key == "kb"))
        if _on_device["lvl1"] != key:
            engine.initialize(ek)  # releases the lvl02 keys, too
            _on_device.update(lvl1=key, lvl02=None)
    return sk


# ------------------------------------------------------------------ cases ----
def _to_gpu(words):
    return torch.from_numpy(np.ascontiguousarray(words).view(np.int32)).cuda()


def _ops(case, rng):
    n = case["count"]
    if case["mix"] == "mixed":
        return rng.choice(np.array(MIX, np.int32), n).astype(np.int32)
    return np.full(n, P.NAND if case["mix"] == "nand" else P.MUX, np.int32)


def _adders(case):
    return circuits.merge([circuits.ripple_carry_adder(case["width"])
                           for _ in range(case["adders"])])


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 77])
    s = {"kind": kind}
    if kind == "gates":
        sk = _load_keys(case["level"], case["key"])
        engine.set_precision(P.INT8_EXACT if case["form"] == "int8" else P.FP64_FFNT)
        n, lvl = case["count"], 1 if case["level"] == 1 else 0
        s["ops"] = _ops(case, rng)
        s["level"] = {0: engine.LVL0, 1: engine.LVL1, 2: engine.LVL02}[case["level"]]
        mux = case["mix"] != "nand"
        s["in"] = [_to_gpu(client.encrypt_bits(sk, rng.integers(0, 2, n).astype(np.uint8), lvl,
                                               seed=seed * 8 + k + 1)) if k < 2 or mux else None
                   for k in range(3)]
        s["out"] = torch.empty_like(s["in"][0])
    elif kind == "circuit":
        sk = _load_keys(1, "kb")
        engine.set_precision(P.FP64_FFNT)
        net = _adders(case)
        ct = client.encrypt_bits(sk, rng.integers(0, 2, net.inputs.size).astype(np.uint8), 1,
                                 seed=seed * 8 + 1)
        wires = np.zeros((net.num_wires, P.TLWE1_WORDS), np.uint32)
        wires[net.inputs] = ct
        s["wires"] = _to_gpu(wires)
        s["circuit"] = engine.Circuit(engine.LVL1, net.num_wires, net.ops, net.in0, net.in1,
                                      net.in2, net.out)
    elif kind == "keyswitch":
        sk = _load_keys(1, "kb")
        s["in"] = _to_gpu(client.encrypt_bits(
            sk, rng.integers(0, 2, case["count"]).astype(np.uint8), 1, seed=seed * 8 + 1))
        s["out"] = torch.empty((case["count"], P.TLWE0_WORDS), dtype=torch.int32, device="cuda")
    else:
        sk = _load_keys(1, "kb")
        q = case["tables"]
        s["luts"] = rng.integers(0, 256, (q, 256)).astype(np.uint8)
        bits = rng.integers(0, 2, q * 8)
        # a pool of encryptions of 0 and of 1; each table takes its eight from it
        pool = _to_gpu(np.stack([client.trgsw_encrypt_g(sk, m, seed=seed * 8 + 1, stream=64 * i,
                                                        l=3, bgbit=6)
                                 for i, m in enumerate([0, 1] * 8)]))
        pick = torch.from_numpy(2 * rng.integers(0, 8, q * 8) + bits).cuda()
        trgsw = pool[pick].contiguous()
        s["trgsw"] = torch.empty((q * 8, 6, 2, 512, 2), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        engine.trgsw_to_fft(engine.GADGET_CB, trgsw, q * 8, s["trgsw"])
        s["out"] = torch.empty((q, 8, P.TLWE1_WORDS), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "gates":
        a, b, c = s["in"]
        engine.gate_batch(s["ops"], s["ops"].size, s["level"], s["out"], a, b, c)
        return s["out"]
    if kind == "circuit":
        s["circuit"].run(s["wires"])
        return s["wires"]
    if kind == "keyswitch":
        engine.identity_keyswitch(s["in"], s["in"].shape[0], s["out"])
        return s["out"]
    engine.lut_eval(s["luts"], s["trgsw"], P.MU32, s["out"])
    return s["out"]


# ------------------------------------------------------------- accounting ----
# operations of one blind rotation: 5 M log2 M per M-point transform and 8 per
# complex multiply-add (FP64 forms), 2 per INT8 product (exact form)
ROTATION = {("fp64", 1, "kb"): 91.5e6, ("fp64", 1, "plain"): 120.5e6,
            ("int8", 1, "kb"): 64.0e9, ("int8", 1, "plain"): 42.7e9,
            ("fp64", 2, "kb"): 349.1e6, ("fp64", 2, "plain"): 459.7e6}
KEY_BYTES = {(1, "kb"): P.BKKB_WORDS * 8, (1, "plain"): P.BK_WORDS * 8,
             (2, "kb"): P.BK2KB_WORDS * 8, (2, "plain"): P.BK2_WORDS * 8}
KSK_BYTES = P.KSK_WORDS * 4
# key switching as it is defined: one 637-word row added per digit
KEYSWITCH = 1024 * 7 * 637


def work(case):
    kind = case["kind"]
    if kind == "gates":
        n = case["count"]
        mux = {"nand": 0.0, "mux": 1.0, "mixed": 1.0 / len(MIX)}[case["mix"]]
        lanes = n * (1 + mux)
        lvl = 2 if case["level"] == 2 else 1
        words = P.TLWE1_WORDS if case["level"] == 1 else P.TLWE0_WORDS
        return {"bytes": 4.0 * words * n * (3 + mux) + KEY_BYTES[lvl, case["key"]] +
                KSK_BYTES * lvl,
                "flops": lanes * (ROTATION[case["form"], lvl, case["key"]] + KEYSWITCH * lvl)}
    if kind == "circuit":
        # three gates of four rotations in all per bit
        bits = case["adders"] * case["width"]
        return {"bytes": 4.0 * P.TLWE1_WORDS * 10 * bits + KEY_BYTES[1, "kb"] + KSK_BYTES,
                "flops": 4.0 * bits * (ROTATION["fp64", 1, "kb"] + KEYSWITCH)}
    if kind == "keyswitch":
        return {"bytes": 4.0 * case["count"] * (P.TLWE1_WORDS + P.TLWE0_WORDS) + KSK_BYTES,
                "flops": float(case["count"]) * KEYSWITCH}
    q = case["tables"]
    # 255 CMUXes per table: six forward and two inverse 512-point transforms
    # and twelve products per bin
    return {"bytes": q * (256.0 + 8 * 6 * 2 * 512 * 16 + 8 * P.TLWE1_WORDS * 4),
            "flops": q * 255.0 * (8 * 5 * 512 * 9 + 12 * 512 * 8)}


def tolerance(case):
    """Every output is a whole number.  The key switches and the exact form are
    integer arithmetic; the FP64 forms at lvl1 round to the exact integer
    result (products below 2^44 in units of 2^-32 against 53 bits), so another
    correct FP64 transform gives the same words.  At lvl2 the last digit of
    the gadget lies below the FP64 rounding, so the same words need the same
    rounding."""
    return "exact"


def exact(case, seed):
    """No floating outputs: the words are compared bit for bit instead."""
    return None
