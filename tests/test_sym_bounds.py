"""The size of generated constraint kernels (csrc/symair.cuh, split_chunks): no
kernel holds more DAG nodes than its bound or, alone, one larger constraint,
and every constraint is folded once. The AIRs have one constraint that reads
many columns, which shares its cells with every other constraint."""
import re

import numpy as np
import pytest

import oracle_ffi as O

GROUP_NODES = 1024  # default bound of a kernel
ADD, NEG = 10, 13


def fingerprint_eval(n, span):
    """n bits, n products of neighbouring bits and a fingerprint column: one
    weighted sum over all bits, sums over `span` bits that overlap by half (0:
    none), and a boolean and a product constraint per bit."""
    def ev(b):
        cols = b.main()[0]
        x, y, f = cols[:n], cols[n:2 * n], cols[2 * n]
        s = x[0] * 3
        for i in range(1, n):
            s = s + x[i] * (i + 3)
        b.assert_zero(s - f)
        for a in range(0, n - span if span else 0, max(1, span // 2)):
            t = x[a] * x[a + 1]
            for i in range(a, a + span - 1):
                t = t + (x[i] * x[i + 1] - y[i]) * 5
            b.assert_zero(t - y[a])
        for i in range(n):
            b.assert_zero(x[i] * (x[i] - 1))
        for i in range(n - 1):
            b.assert_zero(x[i] * x[i + 1] - y[i])
    return ev


def fingerprint_trace(n, h, seed):
    x = np.random.default_rng(seed).integers(0, 2, size=(h, n), dtype=np.uint64)
    t = np.zeros((h, 2 * n + 1), dtype=np.uint64)
    t[:, :n] = x
    t[:, n:2 * n - 1] = x[:, :-1] * x[:, 1:]
    t[:, 2 * n] = x @ np.arange(3, n + 3, dtype=np.uint64)
    return t


def kernel_nodes(src, desc):
    """Operations and cells each generated kernel defines."""
    op = desc.nodes["op"]
    inner = lambda i: op[i] in (1, 2) or ADD <= op[i] <= NEG
    kernels = src[src.index("struct KArgs"):].split("p3g_sym_eval_")[1:]
    return kernels, [sum(inner(int(i)) for i in set(re.findall(r"(?:uint64_t|gl::ef) v(\d+)", k))) for k in kernels]


def constraint_nodes(desc, k):
    seen, st = set(), [int(desc.constraints[k])]
    while st:
        i = st.pop()
        if i in seen:
            continue
        seen.add(i)
        x = desc.nodes[i]
        if ADD <= x["op"] <= NEG:
            st += [int(x["a"])] if x["op"] == NEG else [int(x["a"]), int(x["b"])]
    return sum(desc.nodes[i]["op"] in (1, 2) or desc.nodes[i]["op"] >= ADD for i in seen)


@pytest.mark.parametrize("n,span", [(20, 0), (100, 0), (200, 0), (341, 0), (342, 0), (2000, 0), (120, 40), (400, 130),
                                    (900, 300)])
def test_kernels_stay_within_their_bound(product, n, span):
    desc = product.build_air(fingerprint_eval(n, span), 2 * n + 1)
    src = product.air_source(desc)
    kernels, nodes = kernel_nodes(src, desc)
    largest = max(constraint_nodes(desc, k) for k in range(desc.num_constraints))
    assert max(nodes) <= max(GROUP_NODES, largest)
    # each constraint's power of alpha is read by one kernel's fold
    first = min(int(a) for a in re.findall(r"f0\.mac\(v\d+, __ldg\(K \+ (\d+)\)\)", src))
    folded = sorted((int(a) - first) // 2 for a in re.findall(r"f0\.mac\(v\d+, __ldg\(K \+ (\d+)\)\)", src))
    assert folded == list(range(desc.num_constraints))


@pytest.mark.gpu
@pytest.mark.parametrize("n,span,bound", [(60, 0, 0), (60, 24, 64), (60, 24, 200), (380, 120, 0)])
def test_proof_of_bounded_kernels_matches_oracle(product, n, span, bound):
    desc = product.build_air(fingerprint_eval(n, span), 2 * n + 1)
    t = fingerprint_trace(n, 32, n)
    ctx = product.Context(0)
    try:
        ctx.set_air_chunk_nodes(bound)
        air = product.Air(ctx, desc)
        gpu = product.prove_multi(ctx, product.PcsParams(1, 1, 0, 4, 0, 8, 0), [product.AirWitness(air, t)])
    finally:
        ctx.close()
    pcs = dict(log_blowup=1, log_folding_arity=1, log_final_degree=0, folding_pow_bits=4, deep_pow_bits=0,
               num_queries=8, query_pow_bits=0)
    orc = O.prove(O.default_p2(), pcs, [(O.AIR_SYMBOLIC, t, None, {"sym": desc})])
    assert np.array_equal(gpu.proof.fields, orc["fields"])
    assert np.array_equal(gpu.digest, orc["digest"])
