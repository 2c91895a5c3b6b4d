"""FRI parameters whose last fold is larger than the domain that is left: the
prover and the verifier refuse them (csrc/prover.cuh, fri_rounds_fit); the
parameters beside them still give the oracle's proof."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_h,log_blowup,log_arity,fits", [(3, 1, 3, True), (4, 1, 3, False), (5, 1, 3, True),
                                                             (6, 1, 3, True), (7, 1, 3, False), (5, 1, 2, True),
                                                             (6, 1, 2, True), (5, 2, 3, True), (6, 2, 3, True)])
def test_last_fold(product, gpu_ctx, log_h, log_blowup, log_arity, fits):
    k, t = O.cubic_trace(log_h, 3, 1)
    pcs = product.PcsParams(log_blowup, log_arity, 0, 2, 0, 4, 0)
    wit = product.AirWitness(product.AIR_CUBIC, t, k)
    assert (-(-log_h // log_arity) * log_arity <= log_h + log_blowup) == fits
    if fits:
        out = product.prove_multi(gpu_ctx, pcs, [wit])
        orc = O.prove(O.default_p2(), dict(log_blowup=log_blowup, log_folding_arity=log_arity, log_final_degree=0,
                                           folding_pow_bits=2, deep_pow_bits=0, num_queries=4, query_pow_bits=0),
                      [(O.AIR_CUBIC, t, k)])
        assert np.array_equal(out.proof.fields, orc["fields"])
        assert np.array_equal(out.digest, orc["digest"])
        return
    with pytest.raises(product.P3gError) as e:
        product.prove_multi(gpu_ctx, pcs, [wit])
    assert e.value.status == product.ERR_INVALID
    shape = [product.AirShape(product.AIR_CUBIC, t.shape[0], t.shape[1], k)]
    words = np.zeros(500, dtype=np.uint64)
    r = product.verify_multi(gpu_ctx, pcs, shape, words, words[:160].reshape(-1, 4), words[:12])
    assert r.verdict == 1  # the shape check
