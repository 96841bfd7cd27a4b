"""What is measured: the shard prover's work, case by case.

A prover host holds one context with the resident SRS of its largest shard and
calls, for every shard: the commitments of its trace columns, the layered GKR
proof, and one batched opening; beside them a zerocheck over a shard's tables
and the generic multi-scalar multiplications of the deferred pairing checks.
Shards have 2^8 to 2^22 rows and 4 to 16 columns (even heights only where a
Mercury commitment is involved, which takes no others); column values look
like VM traces (bits, 32-bit words, some full field elements) or, in the worst
case, are uniform field elements.

Every output is a canonical field element, a point encoding or a transcript
state: whole bytes, the same on every run, so they are compared bit for bit
and `exact` has nothing to give.
"""
import math
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "apogee-vm_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import apogee_gpu as A  # noqa: E402
import shard  # noqa: E402
import synth  # noqa: E402

ARTIFACTS = os.path.join(ROOT, "tests", "golden", "artifacts")
DEVICE = "cuda:0"
MAX_LOG = 22                     # the largest shard's rows, and the SRS's powers
TAU = 0x9E3779B97F4A7C15F39CC060  # benchmark-only setup
PRODUCT = 2 * 136                # one 8x32-limb Montgomery product: 136 multiply-adds
FAMILIES = ["add_sub", "jump_branch_slt", "mem_word", "memory_frame_reg", "mul_div", "shift_bitwise"]

_held = {}


def context():
    """The one context a prover process keeps, with the resident SRS."""
    if "ctx" not in _held:
        ctx = A.Context(0)
        ctx.srs_generate(TAU % A.P_R, 1 << MAX_LOG)
        ctx.srs_prepare()
        _held["ctx"] = ctx
    return _held["ctx"]


def base_points():
    """Canonical encodings of some points of the SRS (generic MSM bases)."""
    if "points" not in _held:
        _held["points"] = context().srs_download(1 << 16)
    return _held["points"]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # The smallest shard's commitments: launch and chain latency only.
        {"name": "commit 4x2^8", "kind": "commit", "log": 8, "cols": 4, "values": "mixed"},
        # One uniform 16-variable polynomial from host memory (the plain commit).
        {"name": "commit host 2^16", "kind": "commit_host", "log": 16, "values": "uniform"},
        # The largest shard's commit phase.
        {"name": "commit 16x2^22", "kind": "commit", "log": 22, "cols": 16, "values": "mixed"},
        # A byte column (a lookup multiplicity or range column) in its stored width.
        {"name": "commit narrow u8 2^20", "kind": "narrow", "log": 20, "bits": 8},
        # One block's deferred checks, 207 of 12 entries each, as one generic-base MSM.
        {"name": "msm 2484", "kind": "msm", "n": 2484},
        # The plain method's product sumcheck over the 2^16 commitment's rows.
        {"name": "zerocheck a*b 2^16", "kind": "zerocheck", "log": 16, "arity": 2, "terms": "product"},
        # A gate zerocheck with linear and product terms, an odd number of variables.
        {"name": "zerocheck 4 terms 2^21", "kind": "zerocheck", "log": 21, "arity": 3, "terms": "mixed"},
        # The GKR forward pass and proof of a large synthetic shard circuit.
        {"name": "gkr 10x2^21", "kind": "gkr", "log": 21, "cols": 10},
        # The same over a real family circuit: wide, multiply-heavy gate lists.
        {"name": "gkr add_sub 2^16", "kind": "family", "log": 16, "artifact": "add_sub"},
        # A stacked opening of a middle-sized shard's columns.
        {"name": "open 2x3 stacked 2^14", "kind": "open_stacked", "log": 14, "stacks": 2, "slots": 3, "r": 2},
        # The largest shard's batched opening.
        {"name": "open 16x2^22", "kind": "open", "log": 22, "cols": 16},
        # A whole small shard: commit, transcript, GKR forward and proof, opening.
        {"name": "shard 7x2^12", "kind": "shard", "log": 12, "cols": 7},
    ]


def draw(rng):
    kind = rng.choice(["commit", "commit", "commit_host", "narrow", "msm", "zerocheck", "gkr", "family",
                       "open_stacked", "open", "shard", "shard"])
    if kind == "commit":
        # (Uniform columns cost about three mixed ones: fewer of them at once.)
        values = rng.choice(["mixed", "mixed", "uniform"])
        return {"kind": kind, "log": 2 * rng.randint(4, 11), "cols": rng.randint(1, 16 if values == "mixed" else 4),
                "values": values}
    if kind == "commit_host":
        return {"kind": kind, "log": 2 * rng.randint(4, 10), "values": rng.choice(["mixed", "uniform"])}
    if kind == "narrow":
        return {"kind": kind, "log": 2 * rng.randint(4, 11), "bits": rng.choice([1, 8, 16, 32])}
    if kind == "msm":
        return {"kind": kind, "n": int(math.exp(rng.uniform(math.log(64), math.log(65536))))}
    if kind == "zerocheck":
        return {"kind": kind, "log": rng.randint(8, 22), "arity": rng.randint(2, 5),
                "terms": rng.choice(["product", "mixed"])}
    if kind == "gkr":
        log = rng.randint(8, 21)
        return {"kind": kind, "log": log, "cols": rng.randint(4, 16 if log < 21 else 10)}
    if kind == "family":
        return {"kind": kind, "log": rng.randint(8, 16), "artifact": rng.choice(FAMILIES)}
    if kind == "open_stacked":
        r = rng.randint(1, 3)
        log = 2 * rng.randint(4, 9) + (r & 1)
        return {"kind": kind, "log": log, "stacks": rng.randint(1, 4), "slots": rng.randint(1, 1 << r), "r": r}
    if kind == "open":
        return {"kind": kind, "log": 2 * rng.randint(4, 11), "cols": rng.randint(1, 16)}
    return {"kind": "shard", "log": 2 * rng.randint(4, 9), "cols": rng.randint(4, 16)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _column(log, seed, values="mixed"):
    ctx = context()
    t = synth.device_column(ctx, torch, 1 << log, seed, values, DEVICE)
    ctx.fr_to_mont_device(t.data_ptr(), 1 << log)
    return t


def _columns(case, seed, count=None, values=None):
    return [_column(case["log"], (seed << 8) + j, values or case.get("values", "mixed"))
            for j in range(count or case["cols"])]


def _host_bytes(t):
    return t.cpu().numpy().tobytes()


def _scalars(rng, count):
    return [rng.randrange(A.P_R) for _ in range(count)]


def _transcript(seed):
    return A.transcript_append_scalars(A.transcript_init(), shard.TAG_SHARD_SEED, [seed + 1, seed + 2])


def _gate(terms):
    """A gate's (coefficient, a, b) terms: the product a*b, or one with a
    boolean-style constraint and linear parts over three inputs."""
    if terms == "product":
        return [(1, 0, 1)]
    return [(1, 0, 1), (A.P_R - 1, 2, None), (5, 1, 1), (A.P_R - 7, 0, None)]


def prepare(case, seed):
    rng = random.Random(seed)
    ctx, kind = context(), case["kind"]
    state = {"ctx": ctx, "case": case}
    if kind == "commit":
        state["cols"] = _columns(case, seed)
        state["ptrs"] = [t.data_ptr() for t in state["cols"]]
    elif kind == "commit_host":
        state["evals"] = _host_bytes(_column(case["log"], seed, case["values"]))
    elif kind == "narrow":
        bits, n = case["bits"], 1 << case["log"]
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        state["data"] = torch.randint(0, 256, (max(8, n * bits // 8),), dtype=torch.uint8, device=DEVICE,
                                      generator=g).cpu().numpy().tobytes()
    elif kind == "msm":
        pts, n = base_points(), case["n"]
        at = rng.randrange(len(pts) // 64 - n + 1)
        state["bases"] = pts[64 * at:64 * (at + n)]
        state["scalars"] = A.to_mont_bytes(_scalars(rng, n))
    elif kind == "zerocheck":
        state["terms"] = _gate(case["terms"])
        state["cols"] = _columns(case, seed, max(case["arity"], 3 if case["terms"] == "mixed" else 2), "uniform")
        state["ptrs"] = [t.data_ptr() for t in state["cols"]]
        state["transcript"] = _transcript(seed)
    elif kind in ("gkr", "family"):
        if kind == "gkr":
            state["blob"], count, width, ext = shard.shard_circuit(case["log"], case["cols"]), case["cols"], 0, None
        else:
            state["blob"], count, width = shard.family_circuit(ARTIFACTS, case["artifact"], case["log"])
            ext = shard.statement_challenges()
        g, beta = _scalars(rng, 2)
        state["challenges"] = shard.shard_challenges(g, beta, width, ext)
        state["cols"] = _columns(case, seed, count)
        state["ptrs"] = [t.data_ptr() for t in state["cols"]]
        state["transcript"] = _transcript(seed)
    elif kind == "open":
        state["cols"] = _columns(case, seed)
        state["ptrs"] = [t.data_ptr() for t in state["cols"]]
        state["cms"] = ctx.commit_batch_device(state["ptrs"], case["log"])
        state["u"] = _scalars(rng, case["log"])
        state["transcript"] = _transcript(seed)
    elif kind == "open_stacked":
        state["cols"] = _columns(case, seed, case["stacks"] * case["slots"])
        ptrs = [t.data_ptr() for t in state["cols"]]
        s = case["slots"]
        state["stacks"] = [ptrs[j * s:(j + 1) * s] for j in range(case["stacks"])]
        state["cms"] = [ctx.commit_stack_device(st, case["log"]) for st in state["stacks"]]
        state["u"], state["r"] = _scalars(rng, case["log"]), _scalars(rng, case["r"])
        state["transcript"] = _transcript(seed)
    elif kind == "shard":
        spec = {"index": seed % 4096, "family": seed % shard.FAMILIES, "log_rows": case["log"], "cols": case["cols"]}
        state["cols"] = _columns(case, seed)
        state["shard"] = shard.make_shard(spec, state["cols"])
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _bytes(*parts):
    return torch.frombuffer(bytearray(b"".join(parts)), dtype=torch.uint8)


def _ints(values):
    return b"".join(v.to_bytes(32, "little") for v in values)


def run(state):
    ctx, case, kind = state["ctx"], state["case"], state["case"]["kind"]
    if kind == "commit":
        return _bytes(*ctx.commit_batch_device(state["ptrs"], case["log"]))
    if kind == "commit_host":
        return _bytes(ctx.commit(state["evals"], case["log"]))
    if kind == "narrow":
        return _bytes(ctx.commit_narrow(state["data"], case["bits"], case["log"]))
    if kind == "msm":
        return _bytes(ctx.msm(state["bases"], state["scalars"]))
    if kind == "zerocheck":
        rounds, finals, tr = ctx.prove_zerocheck(state["terms"], state["ptrs"], case["log"], state["transcript"],
                                                 on_device=True)
        return {"rounds": _bytes(*[_ints(r) for r in rounds]), "finals": _bytes(_ints(finals)), "transcript": _bytes(tr)}
    if kind in ("gkr", "family"):
        values = ctx.gkr_forward(state["blob"], state["ptrs"], state["challenges"], on_device=True)
        proof, tr, point = ctx.gkr_prove(state["blob"], values, state["challenges"], state["transcript"],
                                         with_point=True)
        values.free()
        return {"proof": _bytes(_ints(proof)), "transcript": _bytes(tr), "point": _bytes(point)}
    if kind == "open":
        vs, proof, tr = ctx.batch_open(state["ptrs"], case["log"], state["cms"], state["u"], state["transcript"],
                                       on_device=True)
        return {"values": _bytes(_ints(vs)), "proof": _bytes(proof), "transcript": _bytes(tr)}
    if kind == "open_stacked":
        vs, proof, tr = ctx.batch_open_stacked(state["stacks"], case["log"], state["cms"], state["u"], state["r"],
                                               state["transcript"], on_device=True)
        return {"values": _bytes(_ints(vs)), "proof": _bytes(proof), "transcript": _bytes(tr)}
    proof = ctx.prove_shard(state["shard"])
    return {"cms": _bytes(*proof.cms), "gkr": _bytes(_ints(proof.gkr)), "point": _bytes(_ints(proof.point)),
            "values": _bytes(_ints(proof.values)), "opening": _bytes(proof.opening),
            "transcript": _bytes(proof.transcript)}


def exact(case, seed):
    """No output is a rounded number: every one is compared bit for bit."""
    return None


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _msm_products(n, bits=None, mixed=False):
    """Field products of n scalar-point terms: windows as wide as the bucket
    set is worth, six products for each nonzero digit's affine addition."""
    c = max(3, min(20, n.bit_length() - 3))
    full = math.ceil(255 / c)
    if bits:
        digits = math.ceil((bits + 1) / c)
    else:
        digits = 0.125 + 0.6 * math.ceil(33 / c) + 0.15 * full if mixed else full
    return 6 * n * digits


def _sumcheck(n, tables, products):
    """(bytes, products) of a sumcheck over `tables` tables of n entries: each
    read once; every level folded, and `products` a pair at two nodes."""
    return 32 * n * tables, n * (tables + 1) + 2 * n * (products + 1)


def _gkr(n, cols):
    """The synthetic circuit: a row-wise list, then a halving list a variable."""
    b, f = _sumcheck(n, cols, 3 * cols)
    return b, f + 3 * n * cols + _sumcheck(n, 2 * cols, cols)[1] + n * cols


def _open(n, cols):
    b = math.isqrt(n)
    return 32 * n * cols, 2 * n * cols + 4 * n + 2 * _msm_products(n) + 6 * _msm_products(b)


def work(case):
    kind, n = case["kind"], 1 << case["log"] if "log" in case else case["n"]
    if kind == "commit":
        k = case["cols"]
        b, f = 32 * n * k + 64 * n, k * _msm_products(n, mixed=case["values"] == "mixed")
    elif kind == "commit_host":
        b, f = 96 * n, _msm_products(n, mixed=case["values"] == "mixed")
    elif kind == "narrow":
        b, f = 64 * n + n * case["bits"] / 8, _msm_products(n, bits=case["bits"])
    elif kind == "msm":
        b, f = 96 * n, _msm_products(n) + 4 * n
    elif kind == "zerocheck":
        tables = max(case["arity"], 3 if case["terms"] == "mixed" else 2)
        b, f = _sumcheck(n, tables, 1 if case["terms"] == "product" else 4)
    elif kind == "gkr":
        b, f = _gkr(n, case["cols"])
    elif kind == "family":  # about 200 products a row and node in the wide lists
        cols = shard.family_circuit(ARTIFACTS, case["artifact"], case["log"])[1]
        b, f = 32 * n * cols, n * (cols + 3 * 200)
    elif kind == "open":
        b, f = _open(n, case["cols"])
    elif kind == "open_stacked":
        b, f = 32 * n * case["stacks"] * case["slots"], _open(n << case["r"], 1)[1]
    else:
        k = case["cols"]
        parts = [_gkr(n, k), _open(n, k), (64 * n, k * _msm_products(n, mixed=True))]
        b, f = 32 * n * k + 64 * n, sum(p[1] for p in parts)
    return {"bytes": b, "flops": f * PRODUCT}
