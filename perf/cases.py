"""Workloads of this library as a user's program runs them, for timing.

Each case is a dict of plain values; `prepare` makes what such a program holds
before the call (inputs on the GPU, a context, a compiled AIR), `run` is one
pass through the public entry points. All outputs are exact: canonical
Goldilocks words (whole numbers), so two builds must agree bit for bit.

Kinds
  lde      coset_lde of a device matrix (the encode direction of a commit)
  commit   LmcsTree over device matrices, then root and the query openings
  fold     one FRI round's fold
  deep     DEEP openings of committed matrices, then the DEEP quotient
  prove    prove_multi, the whole call
  verify   verify_batch, the other direction of the whole call
"""
import importlib.util
import json
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
DEVICE = 0


def _package():
    if "p3_miden_b200" in sys.modules:
        return sys.modules["p3_miden_b200"]
    pkg = ROOT / "p3-miden_b200"
    spec = importlib.util.spec_from_file_location("p3_miden_b200", pkg / "__init__.py",
                                                  submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["p3_miden_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


P = _package()
SHIFT = 7  # the coset generator of a commitment

# What a program keeps for its lifetime: one context with the saved launch
# shapes (as bench.py applies them) and the compiled symbolic Keccak AIR.
_kept = {}


def _context():
    if "ctx" not in _kept:
        ctx = P.Context(DEVICE)
        table = ROOT / "p3-miden_b200" / "tuning" / "b200.json"
        if table.exists():
            ctx.load_tuning(json.loads(table.read_text()))
        _kept["ctx"] = ctx
    return _kept["ctx"]


def _keccak_air():
    if "air" not in _kept:
        import p3_miden_b200.airs as airs
        _kept["air"] = P.Air(_context(), P.build_air(airs.keccak_eval, airs.KC_NCOLS))
    return _kept["air"]


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A small trace's extension: narrow and short, bound by latency and
        # launches (an aux trace, or a job at the low end of a serving mix).
        {"name": "lde_small", "kind": "lde", "log_h": 12, "width": 16, "log_blowup": 3},
        # One column slab of the 2^18-row Keccak trace.
        {"name": "lde_slab", "kind": "lde", "log_h": 18, "width": 336, "log_blowup": 1},
        # The tallest trace of the lifted workload, with a ragged width: a
        # three-range transform at blowup 8.
        {"name": "lde_tall_ragged", "kind": "lde", "log_h": 20, "width": 37, "log_blowup": 3},
        # A small commitment and its openings (latency-bound tree).
        {"name": "commit_small", "kind": "commit", "log_hs": "11", "widths": "33", "queries": 30},
        # One column slab of the 2^18-row Keccak commitment (2^19 leaves).
        {"name": "commit_slab", "kind": "commit", "log_hs": "19", "widths": "336", "queries": 100},
        # Three matrices of uneven height in one lifted tree.
        {"name": "commit_lifted", "kind": "commit", "log_hs": "13,16,18", "widths": "1024,250,64", "queries": 100},
        # A FRI layer folded at arity 4.
        {"name": "fold_arity4", "kind": "fold", "log_n": 20, "log_arity": 2},
        # The DEEP stage over committed matrices of uneven height.
        {"name": "deep_lifted", "kind": "deep", "log_hs": "13,16,18", "widths": "1024,250,64", "log_blowup": 3},
        # The smallest whole proof: the 42-permutation Keccak example, from a
        # host trace (latency, launches and host work count).
        {"name": "prove_keccak_2e10", "kind": "prove", "air": "keccak", "log_h": 10, "host": True},
        # Three cubic traces lifted to one height, blowup 8, FRI arity 4.
        {"name": "prove_lifted", "kind": "prove", "air": "cubic", "log_hs": "11,13,16", "widths": "512,256,64",
         "log_blowup": 3, "log_arity": 2, "host": False},
        # The plain prover at scale: 10922 Keccak permutations, constraints
        # through the generated kernels, the trace resident on the device.
        {"name": "prove_keccak_2e18", "kind": "prove", "air": "keccak_symbolic", "log_h": 18, "host": False},
        # A server's check of a batch of proofs, some of them damaged.
        {"name": "verify_batch", "kind": "verify", "log_h": 12, "width": 64, "log_blowup": 3, "proofs": 24},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lifted(rng, max_words):
    """One to three matrices in ascending heights, at most max_words in all."""
    n = rng.randint(1, 3)
    hs = sorted(rng.randint(9, 19) for _ in range(n))
    ws = [_log_uniform(rng, 2, max(3, min(1100, max_words // (n << h)))) for h in hs]
    return ",".join(map(str, hs)), ",".join(map(str, ws))


def draw(rng):
    kind = rng.choice(["lde", "lde", "commit", "commit", "fold", "deep", "prove", "prove", "verify"])
    if kind == "lde":
        lb = rng.randint(1, 3)
        log_h = rng.randint(8, 20)
        w = _log_uniform(rng, 2, min(2633, (1 << 28) >> (log_h + lb)))
        return {"kind": kind, "log_h": log_h, "width": w, "log_blowup": lb}
    if kind == "commit":
        hs, ws = _lifted(rng, 1 << 27)
        return {"kind": kind, "log_hs": hs, "widths": ws, "queries": rng.randint(8, 128)}
    if kind == "fold":
        return {"kind": kind, "log_n": rng.randint(10, 23), "log_arity": rng.randint(1, 3)}
    if kind == "deep":
        hs, ws = _lifted(rng, 1 << 27)
        return {"kind": kind, "log_hs": hs, "widths": ws, "log_blowup": rng.randint(1, 3)}
    if kind == "verify":
        return {"kind": kind, "log_h": rng.randint(8, 14), "width": _log_uniform(rng, 16, 256),
                "log_blowup": rng.randint(1, 3), "proofs": _log_uniform(rng, 12, 40)}
    air = rng.choice(["keccak", "keccak_symbolic", "cubic"])
    host = rng.random() < 0.3
    if air != "cubic":
        return {"kind": kind, "air": air, "log_h": rng.randint(8, 16), "host": host, "perms_short": rng.randint(0, 3)}
    n = rng.randint(1, 3)
    hs = sorted(rng.randint(8, 16) for _ in range(n))
    ws = [_log_uniform(rng, 3, min(512, (1 << 23) >> h)) for h in hs]
    lb = rng.randint(1, 3)
    # the folds must land on the final domain: arity 8 needs a blowup of at least 4
    return {"kind": kind, "air": air, "log_hs": ",".join(map(str, hs)), "widths": ",".join(map(str, ws)),
            "log_blowup": lb, "log_arity": rng.randint(1, 3 if lb > 1 else 2), "host": host}


def _ints(text):
    return [int(v) for v in str(text).split(",")]


def _pcs(case):
    """The example's parameters (16 folding PoW bits, 100 queries); blowup and
    arity by case."""
    return P.PcsParams(case.get("log_blowup", 1), case.get("log_arity", 1), 0, 16, 0, 100, 0)


# ------------------------------------------------------------------ inputs
def _uniform(gen, shape):
    """Uniform field elements on the GPU (canonical words in int64 patterns)."""
    t = torch.randint(-(1 << 63), (1 << 63) - 1, shape, dtype=torch.int64, device=f"cuda:{DEVICE}", generator=gen)
    over = (t < 0) & (t > -(1 << 32))  # words in [p, 2^64)
    return torch.where(over, -t, t)


def _field(rng, n=None):
    return rng.integers(0, P.P, size=n, dtype=np.uint64)


def _ef(rng):
    return tuple(int(v) for v in _field(rng, 2))


def _trace_hw(case):
    if case["air"] == "cubic":
        return list(zip(_ints(case["log_hs"]), _ints(case["widths"])))
    return [(case["log_h"], P.KECCAK_NUM_COLS)]


def _host(t):
    return t.cpu().pin_memory()


def _witnesses(case, seed):
    ctx, out = _context(), []
    if case["air"] == "cubic":
        for i, (log_h, w) in enumerate(_trace_hw(case)):
            k, t = P.generate_cubic_trace_device(ctx, log_h, w, seed + 1000 * i)
            out.append(P.AirWitness(P.AIR_CUBIC, _host(t) if case["host"] else t, k))
        return out
    n = (1 << case["log_h"]) // P.KECCAK_ROWS_PER_HASH - case.get("perms_short", 0)
    t = P.generate_keccak_trace_device(ctx, P.to_device(P.keccak_inputs(seed, n), DEVICE), case["log_h"])
    air = _keccak_air() if case["air"] == "keccak_symbolic" else P.AIR_KECCAK
    return [P.AirWitness(air, _host(t) if case["host"] else t)]


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=f"cuda:{DEVICE}")
    gen.manual_seed(seed)
    s = {"case": case, "ctx": ctx}
    if kind == "lde":
        s["trace"] = _uniform(gen, (1 << case["log_h"], case["width"]))
    elif kind in ("commit", "deep"):
        hs, ws = _ints(case["log_hs"]), _ints(case["widths"])
        s["mats"] = [_uniform(gen, (1 << h, w)) for h, w in zip(hs, ws)]
        if kind == "commit":
            s["indices"] = [int(v) for v in rng.choice(1 << hs[-1], size=case["queries"], replace=False)]
        else:
            s["points"] = (_ef(rng), _ef(rng))
            s["alpha"], s["beta"] = _ef(rng), _ef(rng)
    elif kind == "fold":
        s["layer"] = _uniform(gen, (1 << case["log_n"], 2))
        s["beta"] = _ef(rng)
    elif kind == "prove":
        s["pcs"], s["witnesses"] = _pcs(case), _witnesses(case, seed)
    else:  # verify: proofs of the cubic AIR, a quarter of them damaged in one word
        pcs = _pcs(case)
        s["items"] = []
        for i in range(case["proofs"]):
            k, t = P.generate_cubic_trace_device(ctx, case["log_h"], case["width"], seed * 64 + i)
            o = P.prove_single(ctx, pcs, P.AirWitness(P.AIR_CUBIC, t, k))
            fields = o.proof.fields
            if rng.random() < 0.25:
                at = int(rng.integers(0, fields.size))
                fields[at] = (int(fields[at]) + 1) % P.P
            shape = P.AirShape(P.AIR_CUBIC, 1 << case["log_h"], case["width"], k)
            s["items"].append((pcs, [shape], fields, o.proof.commitments, o.digest))
    return s


def _words(a, cap=None):
    """The words of an array; with `cap` zero-padded to that many (openings
    share path digests, so a proof's length depends on its query indices)."""
    a = np.ascontiguousarray(a).reshape(-1).view(np.int64)
    if cap is None:
        return a
    assert a.size <= cap
    out = np.zeros(cap, dtype=np.int64)
    out[:a.size] = a
    return out


def _proof_caps(case):
    """Upper bounds of a proof's field and commitment words."""
    hw, lb, a, q = _trace_hw(case), case.get("log_blowup", 1), case.get("log_arity", 1), 100
    n = hw[-1][0] + lb
    rounds = -(-(n - lb) // a)
    cols = sum(-(-w // 8) * 8 for _, w in hw) + 8 * len(hw) + 8  # main, aux and quotient, aligned
    fields = (4 + q) * cols + rounds * (1 + q * (2 << a)) + (4 << a) + 16
    return fields, 4 * (3 + rounds + q * n * (3 + rounds))


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "lde":
        return P.coset_lde(ctx, s["trace"], case["log_blowup"], SHIFT)
    if kind == "commit":
        tree = P.LmcsTree(ctx, s["mats"], 8)
        rows, siblings = tree.prove_batch(s["indices"])
        return {"root": _words(tree.root()), "rows": _words(rows),
                "siblings": _words(siblings, 4 * len(s["indices"]) * tree.depth)}
    if kind == "fold":
        return P.fri_fold(ctx, s["layer"], case["log_arity"], s["beta"])
    if kind == "deep":
        evals = P.deep_evals(ctx, s["mats"], case["log_blowup"], s["points"])
        q = P.deep_quotient(ctx, s["mats"], case["log_blowup"], 8, s["points"], evals, s["alpha"], s["beta"])
        return {"evals": _words(evals), "quotient": q}
    if kind == "prove":
        o = P.prove_multi(ctx, s["pcs"], s["witnesses"])
        fields, commits = _proof_caps(case)
        return {"digest": _words(o.digest), "fields": _words(o.proof.fields, fields),
                "commitments": _words(o.proof.commitments, commits)}
    verdicts, _ = P.verify_batch(ctx, s["items"])
    return np.array(verdicts, dtype=np.int64)


# -------------------------------------------------------------------- work
# Field operations (a modular multiplication, addition or subtraction each
# count one) of one Poseidon2 permutation: 118 S-boxes of 4 products, 264
# diagonal products, 9 external layers and 22 internal sums.
PERM_OPS = 118 * 4 + 264 + 9 * 60 + 22 * 23


def _perms(mats):
    """Leaf sponge permutations of a lifted tree plus its compressions."""
    return sum((1 << h) * -(-w // 8) for h, w in mats) + (1 << max(h for h, _ in mats))


def _lde_work(log_h, w, lb):
    n_in, B = (1 << log_h) * w, 1 << lb
    # radix-2 butterflies: one product, one sum and one difference per pair
    # and stage, inverse once and forward per coset, and the coset scale
    return 8 * n_in * (1 + B), n_in * (1.5 * log_h * (1 + B) + B)


def _deep_work(mats, lb):
    n = 1 << max(h for h, _ in mats)
    words = sum((1 << h) * w for h, w in mats)
    # openings read the first 1/B of each matrix, the quotient every row
    return 8 * words + 16 * n, words * 4 + 8 * (words >> lb) + 40 * n


def _prove_work(case):
    lb = case.get("log_blowup", 1)
    hw = _trace_hw(case)
    mats = [(h + lb, w) for h, w in hw]
    n = hw[-1][0] + lb
    by, ops = 8 * sum((1 << h) * w for h, w in hw), 0
    for h, w in hw:
        ops += _lde_work(h, w, lb)[1]
        ops += (2 << h) * (w * 8 if case["air"] == "cubic" else 3182 * 6)
    ops += _deep_work(mats, lb)[1]
    ops += PERM_OPS * (_perms(mats) + 4 * (1 << n))
    return by, ops


def work(case):
    kind = case["kind"]
    if kind == "lde":
        by, ops = _lde_work(case["log_h"], case["width"], case["log_blowup"])
    elif kind == "commit":
        mats = list(zip(_ints(case["log_hs"]), _ints(case["widths"])))
        by, ops = 8 * sum((1 << h) * w for h, w in mats), PERM_OPS * _perms(mats)
    elif kind == "fold":
        n = 1 << case["log_n"]
        by, ops = 16 * n + 16 * (n >> case["log_arity"]), 8 * n
    elif kind == "deep":
        by, ops = _deep_work(list(zip(_ints(case["log_hs"]), _ints(case["widths"]))), case["log_blowup"])
    elif kind == "prove":
        by, ops = _prove_work(case)
    else:
        # per query: one row of each matrix, its path and one row and path per FRI round
        n = case["log_h"] + case["log_blowup"]
        per_q = 8 * (case["width"] + 16) + 3 * 32 * n + n * (32 + 16 * n)
        perms_q = case["width"] / 8 + 2 + 3 * n + n * (n + 1) / 2
        by, ops = case["proofs"] * 100 * per_q, case["proofs"] * 100 * perms_q * PERM_OPS
    return {"bytes": float(by), "flops": float(ops)}


def exact(case, seed):
    """Every output is a whole number (a canonical field element, a digest
    word or a verdict) that must come out bit for bit: nothing is rounded."""
    return None
