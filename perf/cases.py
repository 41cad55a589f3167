"""Performance cases of the ring-arithmetic backend: the calls a user's program makes, over the sizes it
makes them at. Every case goes through the public Python entry points (halcuda, ringcuda, trait_ring).

Kinds (a case's "kind"):
  roundtrip   pb_to_crt, a Montgomery product with an operand, crt_to_pb of `count` elements over r factors
  batch       the same for a mixed set of elements of both large fields in one CrtBatch
  hom_mul     BFV ciphertext multiplication of `count` pairs (relinearisation included)
  hom_gal     rotation of `count` ciphertexts by one automorphism
  mod_switch  mod_switch_down of `count` ciphertexts from r to r_out factors
  homcrt      the homomorphic CRT transform of a dBFV ciphertext (baby steps, giant steps, Galois keys)
  dbfv_mul    dBFV ciphertext multiplication
  trait_mul   one ciphertext multiplication issued through the hal::Backend trait methods only
"graph": the call is captured once into a CUDA graph, which a pass replays.

Residues and keys are uniform modulo each factor, as ciphertexts and key-switching keys are. Transforms and
mod-switching work in place or overwrite their input by their nature: a pass continues on what the last one left
(in range: every result is bounded by twice its factor).
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cyclosubfield-dbfv_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import halcuda  # noqa: E402
import ringcuda  # noqa: E402
import trait_ring  # noqa: E402

# field -> (log2 q range, plaintext bits of the ring, an automorphism, conductor): one ring per field for
# every level a program uses, as the serving engine keeps it
RINGS = {
    "field_18": (200, 220, 8, 0, 0),
    "field_192": (400, 420, 8, 0, 0),
    "field_36864": (1100, 1140, 8, 3283177, 8536255),
    "field_49152": (1280, 1310, 8, 20965738, 35297665),
}
DIMS = {"field_18": 18, "field_192": 192, "field_36864": 36864, "field_49152": 49152}
LARGE = ("field_36864", "field_49152")
T = 256
HOMCRT_LOG2_B = 8


def listed():
    return [
        # the smallest call: one element of a unit-test field (launches and host latency are all of it)
        {"name": "roundtrip_f18_r4", "kind": "roundtrip", "field": "field_18", "r": 4, "count": 1},
        # one plaintext or ciphertext element at the level of a 900-bit modulus
        {"name": "roundtrip_f36864_r16", "kind": "roundtrip", "field": "field_36864", "r": 16, "count": 1},
        # a ciphertext (two elements) at the level of a 1280-bit modulus
        {"name": "roundtrip_f49152_r23", "kind": "roundtrip", "field": "field_49152", "r": 23, "count": 2},
        # many elements of uneven levels 4..24 from both fields in one call
        {"name": "batch_128", "kind": "batch", "elements": 128, "mix": 3},
        # one ciphertext multiplication per launch, replayed from a graph (a serving loop's unit)
        {"name": "hom_mul_f36864_r16", "kind": "hom_mul", "field": "field_36864", "r": 16, "count": 1, "graph": True},
        # the same at a low level and without a graph: many short launches
        {"name": "hom_mul_f36864_r5", "kind": "hom_mul", "field": "field_36864", "r": 5, "count": 1, "graph": False},
        # eight pairs in one call
        {"name": "hom_mul_f36864_r16_b8", "kind": "hom_mul", "field": "field_36864", "r": 16, "count": 8, "graph": False},
        # the large field at its full modulus
        {"name": "hom_mul_f49152_r23", "kind": "hom_mul", "field": "field_49152", "r": 23, "count": 1, "graph": False},
        # an odd number of ciphertexts rotated together at an odd level
        {"name": "hom_gal_f49152_r13_b3", "kind": "hom_gal", "field": "field_49152", "r": 13, "count": 3},
        # the linear-transform step of bootstrapping: 13 baby and 5 giant steps over three dBFV digits
        {"name": "homcrt_f49152_r23", "kind": "homcrt", "field": "field_49152", "r": 23, "log2_t": 24, "length": 64},
        # a product of two dBFV ciphertexts of three digits
        {"name": "dbfv_mul_f49152_r16", "kind": "dbfv_mul", "field": "field_49152", "r": 16, "log2_t": 24},
        # what the reference crate runs unchanged on this backend: trait methods only
        {"name": "trait_mul_f36864_r16", "kind": "trait_mul", "field": "field_36864", "r": 16, "count": 1, "graph": True},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("roundtrip", "roundtrip", "batch", "hom_mul", "hom_mul", "hom_gal", "mod_switch", "homcrt",
                       "dbfv_mul", "trait_mul"))
    field = rng.choice(LARGE)
    if kind == "roundtrip":
        field = rng.choice(("field_18", "field_192") + LARGE + LARGE)
        return {"kind": kind, "field": field, "r": rng.randint(1, 4) if field == "field_18" else rng.randint(4, 24) if
                field in LARGE else rng.randint(2, 8), "count": _log_int(rng, 1, 16 if field in LARGE else 200)}
    if kind == "batch":
        return {"kind": kind, "elements": _log_int(rng, 3, 128), "mix": rng.randint(0, 10 ** 6)}
    if kind == "homcrt":
        return {"kind": kind, "field": "field_49152", "r": rng.randint(8, 22), "log2_t": rng.choice((8, 16, 24)),
                "length": rng.randint(20, 64)}
    r = rng.randint(4, 20)
    if kind == "mod_switch":
        return {"kind": kind, "field": field, "r": r, "r_out": rng.randint(2, r - 1), "count": 2 * rng.randint(1, 4)}
    if kind == "dbfv_mul":
        return {"kind": kind, "field": field, "r": rng.randint(6, 16), "log2_t": rng.choice((16, 24))}
    if kind == "trait_mul":
        return {"kind": kind, "field": field, "r": r, "count": 1, "graph": rng.random() < 0.5}
    count = _log_int(rng, 1, 8)
    if kind == "hom_gal":
        return {"kind": kind, "field": field, "r": r, "count": count}
    return {"kind": kind, "field": field, "r": r, "count": count, "graph": rng.random() < 0.5}


# ---------------------------------------------------------------------------------- what a program keeps

_kept = {}


def _backend():
    if "backend" not in _kept:
        _kept["backend"] = halcuda.CudaBackend(0)
    return _kept["backend"]


def _ring(field):
    if field not in _kept:
        lo, hi, t_bits = RINGS[field][:3]
        _kept[field] = ringcuda.RingContext(field, lo, hi, t_bits, backend=_backend())
    return _kept[field]


def _trait(field):
    if ("trait", field) not in _kept:
        _kept["trait", field] = trait_ring.TraitBfv(trait_ring.TraitRing(_ring(field)))
    return _kept["trait", field]


def _residues(R, count, base, gen):
    """[count, r, deg_L', deg_K] residues, uniform in [0, p) for each factor."""
    x = torch.empty(R.shape(count, len(base)), dtype=torch.int64, device="cuda")
    for j, i in enumerate(base):
        x[:, j] = torch.randint(0, R.primes[i], (count, R.dl, R.dk), generator=gen, device="cuda")
    return x


def _dev(x):
    """The library's view of a torch tensor."""
    return halcuda.DeviceTensor(_backend(), x.data_ptr(), tuple(x.shape), tuple(x.stride()), False, owner=x)


class _Array:
    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": t.shape, "typestr": "<i8", "data": (t.ptr, False), "version": 3,
                                         "strides": tuple(8 * s for s in t.strides)}


def _torch(t):
    """A torch tensor over a result that the library allocated."""
    return torch.as_tensor(_Array(t), device="cuda")


def _digits(R, r):
    full = R.initial_len
    return ringcuda.select_digits(math.ceil(full / 4), full)


def _batch_groups(case):
    g = random.Random(case["mix"])
    groups = {}
    for _ in range(case["elements"]):
        k = (g.choice(LARGE), g.randint(4, 24))
        groups[k] = groups.get(k, 0) + 1
    return sorted(groups.items())


def _homcrt_plan(case):
    g, m = RINGS[case["field"]][3:]
    n = case["length"]
    baby = min(range(1, n + 1), key=lambda c: (c + 3 * ((n - 1) // c + 1), c))
    giant = (n - 1) // baby + 1
    return g, baby, giant, sorted({pow(g, j, m) for j in range(1, baby)} | {pow(g, baby, m)})


# ---------------------------------------------------------------------------------- the three functions


def prepare(case, seed):
    be, kind = _backend(), case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": case}
    if kind == "batch":
        items, s["data"] = [], []
        for (field, r), c in _batch_groups(case):
            R, base = _ring(field), list(range(r))
            x, op = _residues(R, c, base, gen), _residues(R, c, base, gen)
            s["data"].append(x)
            items.append((R, _dev(x), _dev(op), base))
        torch.cuda.synchronize()
        s["batch"] = ringcuda.CrtBatch(items, ringcuda.CRT_FORWARD | ringcuda.CRT_MUL | ringcuda.CRT_INVERSE, backend=be)
        return s
    R = s["ring"] = _ring(case["field"])
    r = case["r"]
    base = s["base"] = list(range(r))
    if kind == "roundtrip":
        s["mods"] = R.mods_for(base)
        x, op = _residues(R, case["count"], base, gen), _residues(R, case["count"], base, gen)
        s["data"], s["x"], s["op"] = x, _dev(x), _dev(op)
    elif kind in ("hom_mul", "trait_mul"):
        digits = _digits(R, r)
        ct1, ct2 = (_dev(_residues(R, 2 * case["count"], base, gen)) for _ in range(2))
        rk = _dev(_residues(R, 2 * len(digits), R.initial_base(), gen))
        s["out"] = torch.empty(R.shape(2 * case["count"], r), dtype=torch.int64, device="cuda")
        out = _dev(s["out"])
        mul = R if kind == "hom_mul" else _trait(case["field"])
        s["call"] = lambda: mul.hom_mul(T, ct1, ct2, base, rk, digits, out=out)
        if case["graph"]:
            torch.cuda.synchronize()
            s["call"]()  # the tables of this level, which a capture cannot build
            be.synchronize()
            s["graph"] = halcuda.Graph(be, s["call"])
    elif kind == "hom_gal":
        digits = s["digits"] = _digits(R, r)
        s["ct"] = _dev(_residues(R, 2 * case["count"], base, gen))
        s["key"] = _dev(_residues(R, 2 * len(digits), R.initial_base(), gen))
        s["data"] = torch.empty(R.shape(2 * case["count"], r), dtype=torch.int64, device="cuda")
        s["out"] = _dev(s["data"])
    elif kind == "mod_switch":
        s["x"] = _dev(_residues(R, case["count"], base, gen))
    elif kind == "homcrt":
        g, baby, giant, gs = _homcrt_plan(case)
        digits = _digits(R, r)
        full = R.initial_base()
        key_bytes = 2 * len(digits) * len(full) * R.n * 8
        s["keys"] = ringcuda.Keyset(R, digits, len(full), len(gs) * key_bytes)
        for gg in gs:
            key = _residues(R, 2 * len(digits), full, gen)
            torch.cuda.synchronize()
            s["keys"].add(gg, _dev(key))
            be.synchronize()
        h = random.Random(seed)
        t = 1 << case["log2_t"]
        s["g"], s["coeffs"] = g, [[h.randrange(-t // 2, t // 2) for _ in range(R.dl)] for _ in range(case["length"])]
        s["ct"] = _dev(_residues(R, 2 * ringcuda.dbfv_digits(HOMCRT_LOG2_B, case["log2_t"]), base, gen))
    elif kind == "dbfv_mul":
        s["digits"] = _digits(R, r)
        rows = 2 * ringcuda.dbfv_digits(HOMCRT_LOG2_B, case["log2_t"])
        s["lhs"], s["rhs"] = (_dev(_residues(R, rows, base, gen)) for _ in range(2))
        s["rk"] = _dev(_residues(R, 2 * len(s["digits"]), R.initial_base(), gen))
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        s["batch"].run()
        return s["data"]
    R, base = s["ring"], s["base"]
    if kind == "roundtrip":
        R.pb_to_crt(s["x"], base)
        R.backend.hal_mul_mont64(s["x"], s["op"], s["mods"])
        R.crt_to_pb(s["x"], base)
        return s["data"]
    if kind in ("hom_mul", "trait_mul"):
        if case["graph"]:
            s["graph"].launch()
        else:
            s["call"]()
        return s["out"]
    if kind == "hom_gal":
        R.hom_gal_batch(s["ct"], base, RINGS[case["field"]][3], s["key"], s["digits"], out=s["out"])
        return s["data"]
    if kind == "mod_switch":
        return _torch(R.mod_switch_down(s["x"], base, case["r_out"]))
    if kind == "homcrt":
        return _torch(ringcuda.dbfv_hom_cyclic_transform(R, HOMCRT_LOG2_B, case["log2_t"], s["g"], s["coeffs"], s["ct"],
                                                         base, s["keys"]))
    return _torch(ringcuda.dbfv_hom_mul(R, HOMCRT_LOG2_B, case["log2_t"], s["lhs"], s["rhs"], base, s["rk"], s["digits"]))


def work(case):
    """bytes: inputs, keys and results once each. flops: two for each exact modular product of 64-bit words (a
    multiplication and an addition) that the transforms, base conversions and key switches consist of."""
    kind = case["kind"]
    # products per residue of one transform: a radix-2 stage 1/2, a radix-3 stage 2, both directions, two kernels
    per = {"field_18": 14, "field_192": 18, "field_36864": 22, "field_49152": 20}
    if kind == "batch":
        res = [(f, c * r * DIMS[f]) for (f, r), c in _batch_groups(case)]
        return {"bytes": 24 * sum(n for _, n in res), "flops": 2 * sum((2 * per[f] + 1) * n for f, n in res)}
    field, r = case["field"], case["r"]
    n, p = DIMS[field], per[field]
    c = case.get("count", 1)
    if kind == "roundtrip":
        return {"bytes": 24 * c * r * n, "flops": 2 * (2 * p + 1) * c * r * n}
    d = math.ceil(r / 4)  # gadget digits that reach this level
    key = 2 * d * r  # rows of a key-switching key
    switch = (d * r * p + r * r + 2 * d * r) * n  # decomposition, its transforms, the inner product
    ext = r + 2  # rows of the extension base
    mul = ((4 * r + 4 * ext + 3 * (r + ext) + 2 * r) * p + 4 * r * ext + 4 * (r + ext) + 3 * r * ext) * n + switch
    if kind in ("hom_mul", "trait_mul"):
        return {"bytes": 8 * n * (c * 6 * r + key), "flops": 2 * c * mul}
    if kind == "hom_gal":
        return {"bytes": 8 * n * (c * 4 * r + key), "flops": 2 * c * (r * p * n + switch)}
    if kind == "mod_switch":
        return {"bytes": 8 * n * c * (r + case["r_out"]), "flops": 2 * n * c * (r - case["r_out"]) * case["r_out"]}
    dig = (case["log2_t"] - 1) // HOMCRT_LOG2_B + 1
    if kind == "dbfv_mul":
        pairs = dig * (dig + 1) // 2
        lift = ((4 * r + 4 * ext) * p + 4 * r * ext) * n * dig
        back = ((3 * (r + ext) + 2 * r) * p + 3 * r * ext) * n * dig + dig * switch
        return {"bytes": 8 * n * (6 * dig * r + key), "flops": 2 * (lift + 4 * pairs * (r + ext) * n + back)}
    _, baby, giant, gs = _homcrt_plan(case)
    steps = dig * ((2 * r * p + switch) + (baby - 1) * 2 * d * r * n + (giant - 1) * (r * p * n + switch))
    giants = giant * baby * dig * (dig + 1) * r * n
    return {"bytes": 8 * n * (4 * dig * r + len(gs) * key), "flops": 2 * (steps + giants)}


def exact(case, seed):
    """Every output is a whole number, which has to stay equal."""
    return None
