"""Performance cases of the CKKS evaluation core, through its Python entry points.

A case is one call (or one short chain of calls) that an encrypted program
makes, at one set of parameters: `logn` (ring dimension), `limbs` (ciphertext
moduli, the first 60-bit, the others of `bits` bits), `dnum` (key-switching
digits) and `level` (limbs in use minus one).  Ciphertexts come from the
library's seeded generator (residues of a ciphertext are uniform), except
where slots are decrypted; those are real encryptions.

A context with its keys, and the plaintext matrix of a linear transform, are
made once per parameter set and kept, as a program keeps them; every
prepare() draws its own inputs.  Evaluation results are returned as device
residues, (2, limbs, N) 64-bit words per ciphertext.
"""
import math

import numpy as np
import torch

import pyfideslib_b200 as fides
from pyfideslib_b200._capi import check, lib, u64p

_CONTEXTS = {}

BOOT_LIMBS = 30


def listed():
    return [
        # the smallest call a program makes: one addition in a small ring
        {"name": "add_n12", "kind": "add", "logn": 12, "limbs": 10, "dnum": 3, "bits": 50, "level": 3},
        # product and rescale of a shallow circuit in a small ring: launches and latency count
        {"name": "mult_n13", "kind": "mult", "logn": 13, "limbs": 7, "dnum": 3, "bits": 50, "level": 5},
        # plaintext weights, a scalar factor and a constant (one step of a linear layer) on a 59-bit chain
        {"name": "affine_n14", "kind": "affine", "logn": 14, "limbs": 11, "dnum": 3, "bits": 59, "level": 10},
        # client side: encode + encrypt, then decrypt + decode
        {"name": "client_n15", "kind": "client", "logn": 15, "limbs": 13, "dnum": 3, "bits": 50, "level": 12},
        # one rotation on a 59-bit chain, four digits, an odd level
        {"name": "rotate_n15", "kind": "rotate", "logn": 15, "limbs": 21, "dnum": 4, "bits": 59, "level": 16},
        # plain RNS polynomial product (two forward transforms, one inverse), all 30 limbs
        {"name": "polymul_n16", "kind": "polymul", "logn": 16, "limbs": 30, "dnum": 3, "bits": 50, "level": 29},
        # one product at the top level of the 30-limb chain, as a program without batching makes it
        {"name": "mult_n16", "kind": "mult", "logn": 16, "limbs": 30, "dnum": 3, "bits": 50, "level": 29},
        # the batched headline: 32 independent products at the top level
        {"name": "mult_batch_n16", "kind": "mult_batch", "logn": 16, "limbs": 30, "dnum": 3, "bits": 50, "level": 29,
         "count": 32, "spread": 0},
        # products and rotations of pairs at uneven levels, captured once and replayed
        {"name": "plan_n16", "kind": "plan", "logn": 16, "limbs": 30, "dnum": 3, "bits": 50, "level": 29, "count": 21,
         "spread": 25},
        # 32 hoisted rotations of one ciphertext, 20 limbs of 40 bits
        {"name": "hoist_n16", "kind": "hoist", "logn": 16, "limbs": 20, "dnum": 3, "bits": 40, "level": 19,
         "count": 32},
        # a 64-diagonal plaintext matrix by baby-step giant-step, same chain
        {"name": "transform_n16", "kind": "transform", "logn": 16, "limbs": 20, "dnum": 3, "bits": 40, "level": 19,
         "count": 64},
        # a full-packing bootstrap and the decryption of its result: the largest call
        {"name": "boot_n16", "kind": "boot", "logn": 16, "limbs": BOOT_LIMBS, "dnum": 3, "bits": 50, "level": 0,
         "slots": 1 << 15},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# limbs in use by ring dimension, small parameter sets to the 30-limb chain
_MOST_LIMBS = {12: 10, 13: 12, 14: 16, 15: 24, 16: 30}


def draw(rng):
    kind = rng.choice(["add", "affine", "client", "polymul", "mult", "mult", "mult_batch", "mult_batch", "plan",
                       "rotate", "rotate", "hoist", "transform", "boot"])
    logn = rng.randint(12, 16)
    if kind == "boot":
        logn = rng.randint(12, 15)
        return {"kind": kind, "logn": logn, "limbs": BOOT_LIMBS, "dnum": 3, "bits": 50, "level": rng.randint(0, 3),
                "slots": 1 << rng.randint(5, logn - 1)}
    limbs = _log_int(rng, 4, _MOST_LIMBS[logn])
    dnum = rng.choice([2, 3, 3, 4])
    bits = rng.choice([40, 50, 50, 59])
    level = rng.randint(limbs // 2, limbs - 1) if rng.random() < 0.8 else rng.randint(2, limbs - 1)
    c = {"kind": kind, "logn": logn, "limbs": limbs, "dnum": dnum, "bits": bits, "level": level}
    if kind in ("mult_batch", "plan"):
        c["count"] = _log_int(rng, 2, 32 if kind == "mult_batch" else 16)
        c["spread"] = rng.randint(0, level - 1)
    elif kind in ("hoist", "transform"):
        c["count"] = _log_int(rng, 2, 32 if kind == "hoist" else 48)
    return c


# ---------------------------------------------------------------------------
# contexts
# ---------------------------------------------------------------------------
class _Context:
    def __init__(self, case):
        boot = case["kind"] == "boot"
        self.cc = fides.CryptoContext(log_n=case["logn"], num_q=case["limbs"], dnum=case["dnum"],
                                      qi_bits=case["bits"])
        self.sk = self.cc.KeyGen(seed=101, hamming_weight=32 if boot else 192)
        self.cc.EvalMultKeyGen(self.sk)
        self.rotations = set()
        self.matrices = {}
        if boot:
            budget = 3 if case["slots"] >= 1 << 12 else 2
            self.cc.EvalBootstrapSetup(level_budget=(budget, budget), slots=case["slots"])
            self.cc.EvalBootstrapKeyGen(self.sk, slots=case["slots"])

    def need_rotations(self, indices):
        for r in indices:
            if r not in self.rotations:
                self.cc.EvalRotateKeyGen(self.sk, [r], seed=1000 + (r % self.cc.N))
                self.rotations.add(r)

    def matrix(self, level, count):
        """`count` plaintext diagonals (model weights: the same for every input)."""
        if (level, count) not in self.matrices:
            rng = np.random.default_rng(5 * count + level)
            pts = []
            for _ in range(count):
                m = np.stack([rng.integers(0, q, self.cc.N, dtype=np.uint64) for q in self.cc.q[:level + 1]])
                h = fides._capi.vp()
                check(lib.fides_pt_upload(self.cc._h, m.ctypes.data_as(u64p), level, self.cc.scale, 1,
                                          self.cc.N // 2, h), self.cc._h)
                self.cc.Synchronize()
                pts.append(fides.Plaintext(self.cc, h.value, None, self.cc.N // 2))
            self.matrices[(level, count)] = pts
        return self.matrices[(level, count)]


def _context(case):
    key = tuple(case[k] for k in ("logn", "limbs", "dnum", "bits"))
    if case["kind"] == "boot":  # its keys belong to a sparse secret and one slot count
        key += (case["slots"],)
    if key not in _CONTEXTS:
        _CONTEXTS[key] = _Context(case)
    return _CONTEXTS[key]


# ---------------------------------------------------------------------------
# device residues of a ciphertext as a tensor (a view, no copy)
# ---------------------------------------------------------------------------
class _View:
    def __init__(self, ct, p0, p1, n, ring):
        self.ct = ct  # the tensor keeps its ciphertext alive
        self.__cuda_array_interface__ = {"shape": (2, n, ring), "strides": (p1 - p0, 8 * ring, 8), "typestr": "<i8",
                                         "data": (p0, False), "version": 2}


def _residues(state, ct, n):
    p0, p1 = u64p(), u64p()
    check(lib.fides_ct_device_ptrs(ct._h, p0, p1))
    vp = fides._capi.C.c_void_p
    key = (fides._capi.C.cast(p0, vp).value, fides._capi.C.cast(p1, vp).value, n)
    views = state["views"]
    view = views.get(key)
    if view is None:
        view = torch.as_tensor(_View(ct, *key, state["cc"].N), device="cuda")
        if state["case"]["kind"] != "hoist":  # which makes new ciphertexts on every call
            views[key] = view
    return view


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _levels(case, seed):
    """Levels of a batch: the case's level, down by up to `spread`."""
    rng = np.random.default_rng(7919 + case["count"])
    down = rng.integers(0, case["spread"] + 1, case["count"])
    return [case["level"] - int(d) for d in down]


def _hoisted_indices(case):
    half = 1 << (case["logn"] - 1)
    ks = [s * (1 << k) for k in range(case["logn"] - 1) for s in (1, -1)] + list(range(3, half, 2))
    out = []
    for r in ks:
        if r % half and r not in out:
            out.append(r)
        if len(out) == case["count"]:
            break
    return out


def _slots(case, seed):
    n = case.get("slots") or 1 << (case["logn"] - 1)
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)


def prepare(case, seed):
    x = _context(case)
    cc, kind, lv = x.cc, case["kind"], case["level"]
    s = {"case": case, "cc": cc, "x": x, "views": {}}

    def ct(i, level=lv):
        return cc.random_ct(level, (seed % (1 << 40)) * 1024 + i)

    if kind in ("add", "mult"):
        s["a"], s["b"], s["out"] = ct(0), ct(1), fides.Ciphertext(cc)
    elif kind == "affine":
        s["a"], s["t"], s["out"] = ct(0), fides.Ciphertext(cc), fides.Ciphertext(cc)
        s["w"] = cc.MakeCKKSPackedPlaintext(_slots(case, seed), level=lv)
    elif kind in ("mult_batch", "plan"):
        s["levels"] = _levels(case, seed)
        s["a"] = [ct(2 * i, v) for i, v in enumerate(s["levels"])]
        s["b"] = [ct(2 * i + 1, v) for i, v in enumerate(s["levels"])]
        if kind == "plan":
            half = 1 << (case["logn"] - 1)
            idx = [1 + (2654435761 * (i + 1)) % (half - 1) for i in range(case["count"])]
            x.need_rotations(idx)
            s["plan"], s["outs"] = cc.plan_hmult_rotate(s["a"], s["b"], idx, rescale=True)
        else:
            s["outs"] = [fides.Ciphertext(cc) for _ in s["levels"]]
    elif kind == "rotate":
        s["a"], s["out"], s["index"] = ct(0), fides.Ciphertext(cc), 17
        x.need_rotations([17])
    elif kind == "hoist":
        s["a"], s["idx"] = ct(0), _hoisted_indices(case)
        x.need_rotations(s["idx"])
    elif kind == "transform":
        s["a"], s["out"] = ct(0), fides.Ciphertext(cc)
        s["offsets"] = list(range(case["count"]))
        s["bstep"] = 1 << max(0, round(math.log2(math.sqrt(case["count"]))))
        x.need_rotations(cc.linear_transform_rotations(s["offsets"], s["bstep"]))
        s["pts"] = x.matrix(lv, case["count"])
    elif kind == "polymul":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        n = lv + 1
        for name in ("a", "b"):
            s[name] = torch.stack([torch.randint(0, q, (cc.N,), generator=g, device="cuda", dtype=torch.int64)
                                   for q in cc.q[:n]])
        for name in ("c", "an", "bn"):
            s[name] = torch.empty_like(s["a"])
    elif kind == "client":
        s["v"], s["seed"] = _slots(case, seed), seed % (1 << 40) + 1
    elif kind == "boot":
        s["a"] = cc.Encrypt(x.sk, _slots(case, seed), slots=case["slots"], level=lv, seed=seed % (1 << 40) + 1)
        s["out"] = fides.Ciphertext(cc)
    return s


def run(s):
    case, cc = s["case"], s["cc"]
    kind, lv = case["kind"], case["level"]
    if kind == "add":
        return _residues(s, cc.EvalAdd(s["a"], s["b"], out=s["out"]), lv + 1)
    if kind == "mult":
        return _residues(s, cc.EvalMult(s["a"], s["b"], rescale=True, out=s["out"]), lv)
    if kind == "affine":
        t = cc.EvalMult(s["a"], s["w"], rescale=True, out=s["t"])
        t = cc.EvalMult(t, 0.75, rescale=True, out=s["t"])
        return _residues(s, cc.EvalAdd(t, 0.25, out=s["out"]), lv - 1)
    if kind == "mult_batch":
        outs = cc.EvalMultBatch(s["a"], s["b"], rescale=True, outs=s["outs"])
        return [_residues(s, o, v) for o, v in zip(outs, s["levels"])]
    if kind == "plan":
        s["plan"].launch()
        return [_residues(s, o, v) for o, v in zip(s["outs"], s["levels"])]
    if kind == "rotate":
        return _residues(s, cc.EvalRotate(s["a"], s["index"], out=s["out"]), lv + 1)
    if kind == "hoist":
        s["outs"] = cc.EvalFastRotation(s["a"], s["idx"])
        return [_residues(s, o, lv + 1) for o in s["outs"]]
    if kind == "transform":
        cc.EvalLinearTransform(s["a"], s["offsets"], s["pts"], s["bstep"], rescale=True, out=s["out"])
        return _residues(s, s["out"], lv)
    if kind == "polymul":
        cc.polymul(*(s[k].data_ptr() for k in ("a", "b", "c", "an", "bn")), 0, lv + 1)
        return s["c"]
    if kind == "client":
        ct = cc.Encrypt(s["x"].sk, s["v"], level=lv, seed=s["seed"])
        return cc.Decrypt(s["x"].sk, ct)
    ct = cc.EvalBootstrap(s["a"], out=s["out"])
    return cc.Decrypt(s["x"].sk, ct, slots=case["slots"])


def exact(case, seed):
    # residues are whole numbers; slots that come back decrypted are the message
    if case["kind"] in ("client", "boot"):
        return _slots(case, seed)
    return None


# ---------------------------------------------------------------------------
# compulsory work: bytes of inputs, keys and outputs once; operations are
# modular products, additions and subtractions
# ---------------------------------------------------------------------------
def _special(case):
    alpha = -(-case["limbs"] // case["dnum"])
    widest = 60 + (alpha - 1) * case["bits"]
    return (widest + 58) // 59


def _transform_ops(case, limbs):
    return limbs * 3 * (1 << case["logn"]) * case["logn"] / 2


def _keyswitch(case, level):
    """(operations of ModUp, of inner product + ModDown, limbs of one key)."""
    n, k, ring = level + 1, _special(case), 1 << case["logn"]
    alpha = -(-case["limbs"] // case["dnum"])
    digits = [min(alpha, n - lo) for lo in range(0, n, alpha)]
    up = _transform_ops(case, n) + sum(_transform_ops(case, n - d + k) + 2 * ring * d * (n - d + k) for d in digits)
    down = 4 * ring * len(digits) * (n + k) + 2 * (_transform_ops(case, k + n) + 2 * ring * k * n)
    return up, down, 2 * len(digits) * (n + k)


def work(case):
    kind, lv, ring = case["kind"], case["level"], 1 << case["logn"]
    n, limb = lv + 1, 8 << case["logn"]
    up, down, key = _keyswitch(case, lv)

    def mult(level):
        u, d, _ = _keyswitch(case, level)
        return u + d + 5 * ring * (level + 1) + _transform_ops(case, 2), 4 * (level + 1) + 2 * level

    if kind == "add":
        return {"bytes": 6 * n * limb, "flops": 2 * n * ring}
    if kind == "affine":
        ops = 2 * (2 * n * ring + _transform_ops(case, 2 * n)) + n * ring
        return {"bytes": (3 * n + 2 * (n - 2)) * limb, "flops": ops}
    if kind == "client":
        fft = 2 * 10 * ring * case["logn"] / 2
        return {"bytes": 2 * n * limb + 16 * ring, "flops": fft + _transform_ops(case, 2 * n + 3)}
    if kind == "polymul":
        return {"bytes": 3 * n * limb, "flops": _transform_ops(case, 3 * n) + n * ring}
    if kind == "mult":
        ops, limbs = mult(lv)
        return {"bytes": (limbs + key) * limb, "flops": ops}
    if kind in ("mult_batch", "plan"):
        ops, limbs = 0, key
        for v in _levels(case, 0):
            o, m = mult(v)
            ops, limbs = ops + o, limbs + m
            if kind == "plan":
                u, d, k = _keyswitch(case, v - 1) if v > 1 else _keyswitch(case, 0)
                ops, limbs = ops + u + d, limbs + k // 2
        return {"bytes": limbs * limb, "flops": ops}
    if kind == "rotate":
        return {"bytes": (4 * n + key // 2) * limb, "flops": up + down}
    if kind == "hoist":
        return {"bytes": (2 * n + case["count"] * (2 * n + key // 2)) * limb, "flops": up + case["count"] * down}
    if kind == "transform":
        c = case["count"]
        b = 1 << max(0, round(math.log2(math.sqrt(c))))
        g = -(-c // b)
        ops = up + (b - 1) * down + (g - 1) * (up + down) + 4 * c * n * ring + _transform_ops(case, 2 * n)
        return {"bytes": ((c + 4) * n + (b + g - 2) * (key // 2)) * limb, "flops": ops}
    # bootstrap: about thirty key switches spread over the levels, and the
    # diagonals of six transforms
    top = case["limbs"] - 1
    u, d, k = _keyswitch(case, top * 2 // 3)
    return {"bytes": (60 * top + 40 * (k // 2)) * limb, "flops": 60 * (u + d)}
