"""Bounded waits of the tensor-core hash kernels (csrc/p2tc.cuh, collect): with
no time allowed every wait gives up, the launch ends by itself and the call
returns ERR_TIMEOUT; the next call on the same context is unaffected."""
import numpy as np
import pytest

import oracle_ffi as O

P = O.P


def test_wait_bound_is_checked(product):
    assert product.lib().p3g_ctx_set_hash_wait(None, 0) == product.ERR_INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(1 << 15, 25)],                  # one class, one chunk and more
                                    [(1 << 15, 9), (1 << 17, 8)],     # carried states, tensor-core levels
                                    [(1 << 18, 4)]])                  # several rounds per CTA
def test_tree_after_a_wait_that_gave_up(product, shapes):
    rng = np.random.default_rng(len(shapes))
    mats = [rng.integers(0, P, size=s, dtype=np.uint64) for s in shapes]
    dev = [product.to_device(m) for m in mats]
    ctx = product.Context(0)
    try:
        ctx.set_hash_wait(0)
        for _ in range(2):
            with pytest.raises(product.P3gError) as e:
                product.LmcsTree(ctx, dev, 8)
            assert e.value.status == product.ERR_TIMEOUT
        ctx.set_hash_wait(10 ** 8)
        got = product.LmcsTree(ctx, dev, 8).root()
        with pytest.raises(product.P3gError):
            ctx.set_hash_wait(10 ** 8 + 1)
    finally:
        ctx.close()
    assert np.array_equal(got, O.OracleTree(O.default_p2(), mats, 8).root())


@pytest.mark.gpu
def test_proof_after_a_wait_that_gave_up(product):
    k, t = O.cubic_trace(14, 9, 3)  # 2^15 leaves
    pcs = product.PcsParams(1, 1, 0, 4, 0, 8, 0)
    ctx = product.Context(0)
    try:
        want = product.prove_multi(ctx, pcs, [product.AirWitness(product.AIR_CUBIC, t, k)])
        ctx.set_hash_wait(0)
        with pytest.raises(product.P3gError) as e:
            product.prove_multi(ctx, pcs, [product.AirWitness(product.AIR_CUBIC, t, k)])
        assert e.value.status == product.ERR_TIMEOUT
        ctx.set_hash_wait(10 ** 8)
        got = product.prove_multi(ctx, pcs, [product.AirWitness(product.AIR_CUBIC, t, k)])
    finally:
        ctx.close()
    assert np.array_equal(got.proof.fields, want.proof.fields)
    assert np.array_equal(got.digest, want.digest)
