"""Large classes and levels hashed by one thread per state (csrc/merkle.cuh,
leaf_class_kernel and compress_kernel), which a Poseidon2 table outside the
range of the tensor cores' byte tables takes: bit for bit against the oracle,
and a proof with column-major copies equal to the tensor cores'."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P


@pytest.fixture
def thread_ctx(product):
    ctx = product.Context(0)
    ctx.set_tensor_hash(False)
    yield ctx
    ctx.close()


@pytest.mark.parametrize("shapes,alignment", [([(1 << 15, 9)], 8), ([(1 << 12, 5), (1 << 16, 16), (1 << 16, 3)], 1),
                                              ([(1 << 15, 1), (1 << 17, 8)], 8), ([(1 << 18, 4)], 1)])
def test_trees_match_oracle(product, thread_ctx, shapes, alignment):
    rng = np.random.default_rng(len(shapes))
    mats = [rng.integers(0, P, size=s, dtype=np.uint64) for s in shapes]
    mats[-1][::3] = P - 1
    got = product.LmcsTree(thread_ctx, [product.to_device(m) for m in mats], alignment)
    want = O.OracleTree(O.default_p2(), mats, alignment)
    assert np.array_equal(got.root(), want.root())
    for l in (0, 1, 2):
        assert np.array_equal(got.layer(l), want.layer(l))


def test_proof_equals_the_tensor_cores(product, gpu_ctx, thread_ctx):
    import p3_miden_b200.airs as airs
    t = product.generate_keccak_trace(product.keccak_inputs(2, 682))  # 2^14 rows, 2^15 leaves
    pcs = product.PcsParams(1, 1, 0, 4, 0, 8, 0)
    out = []
    for ctx in (gpu_ctx, thread_ctx):
        air = product.Air(ctx, product.build_air(airs.keccak_eval, airs.KC_NCOLS))
        out.append(product.prove_multi(ctx, pcs, [product.AirWitness(air, t)]))
    assert np.array_equal(out[0].proof.fields, out[1].proof.fields)
    assert np.array_equal(out[0].digest, out[1].digest)
