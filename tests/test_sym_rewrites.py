"""Rewrites of the generated constraint kernels that meet (csrc/symair.cuh): the
operands of (a + b) - (c + c) are themselves sums that only it reads, which
alone would be links of a chain."""
import numpy as np
import pytest

import oracle_ffi as O


def eval_form(form):
    def ev(b):
        x = b.main()[0]
        a, c = x[0], x[3]
        if "a" in form:
            a = x[0] + x[1] - x[2]
        if "n" in form:
            a = -a
        if "c" in form:
            c = x[3] - x[4]
        y = (a + x[5]) - (c + c)
        if "l" in form:  # read by another link
            y = y + x[6] + x[7]
        b.assert_zero(y * x[1] if "m" in form else y)
    return ev


FORMS = ["a", "n", "c", "an", "ac", "acl", "acm", "nclm"]


@pytest.mark.parametrize("form", FORMS)
def test_kernel_compiles(product, form):
    assert product.air_compile_check(product.build_air(eval_form(form), 8)) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
def test_proof_matches_oracle(product, gpu_ctx, form):
    desc = product.build_air(eval_form(form), 8)
    t = np.random.default_rng(len(form)).integers(0, O.P, size=(16, 8), dtype=np.uint64)
    t[::3] = O.P - 1
    air = product.Air(gpu_ctx, desc)
    gpu = product.prove_multi(gpu_ctx, product.PcsParams(1, 1, 0, 2, 0, 6, 0), [product.AirWitness(air, t)])
    pcs = dict(log_blowup=1, log_folding_arity=1, log_final_degree=0, folding_pow_bits=2, deep_pow_bits=0,
               num_queries=6, query_pow_bits=0)
    orc = O.prove(O.default_p2(), pcs, [(O.AIR_SYMBOLIC, t, None, {"sym": desc})])
    assert np.array_equal(gpu.proof.fields, orc["fields"])
    assert np.array_equal(gpu.digest, orc["digest"])
