"""Batch verification of more proofs than a grid's y dimension has blocks
(csrc/verifier.cuh, deep_kernel): small proofs, a few of them perturbed on
both sides of 2^16, each with the verdict of the single call."""
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P


@pytest.mark.parametrize("n", [65535, 65536, 65540])
def test_batch_of_2_16_proofs(product, gpu_ctx, n):
    k, t = O.cubic_trace(2, 2, 5)
    pcs = product.PcsParams(1, 1, 0, 0, 0, 5, 0)  # five queries: two blocks of warps
    out = product.prove_multi(gpu_ctx, pcs, [product.AirWitness(product.AIR_CUBIC, t, k)])
    shapes = [product.AirShape(O.AIR_CUBIC, t.shape[0], t.shape[1], k)]
    f, c, d = out.proof.fields, out.proof.commitments, out.digest
    row, sibling = f.copy(), c.copy()
    row[-3] = (int(row[-3]) + 1) % P
    sibling[-1, 0] = (int(sibling[-1, 0]) + 1) % P
    variants = [(f, c, d), (row, c, d), (f, sibling, d)]
    single = [product.verify_multi(gpu_ctx, pcs, shapes, *v).verdict for v in variants]
    assert single[0] == 0 and single[1] != 0 and single[2] != 0
    which = {0: 1, 3: 2, 65533: 1, 65534: 2, n - 1: 1}
    got, _ = product.verify_batch(gpu_ctx, [(pcs, shapes, *variants[which.get(i, 0)]) for i in range(n)])
    assert got == [single[which.get(i, 0)] for i in range(n)]
