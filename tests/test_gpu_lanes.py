"""Kernels whose lanes follow the size: DEEP row sums by matrix width
(csrc/deep.cuh) against the CPU oracle, and the hashes of batch verification
by the number of openings in the batch (csrc/verifier.cuh) against the single
call."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P


# widths on both sides of each lane count, and the coefficients' block of 1024
@pytest.mark.parametrize("widths,alignment", [([15, 16], 8), ([17, 63], 1), ([64, 65], 8), ([127, 128], 8),
                                              ([129, 255], 1), ([256, 257], 8), ([512, 511], 1), ([3, 1030], 8)])
@pytest.mark.parametrize("kind", ["random", "top"])
def test_deep_of_every_width(product, gpu_ctx, widths, alignment, kind):
    rng = np.random.default_rng(sum(widths))
    lb, hs = 1, [8, 64]  # fewer rows than a warp holds, and more
    word = lambda: int(rng.integers(0, P, dtype=np.uint64)) if kind == "random" else P - 1
    mats = []
    for h, w in zip(hs, widths):
        t = rng.integers(0, P, size=(h >> lb, w), dtype=np.uint64)
        if kind == "top":
            t[:] = P - 1  # a constant column: its extension is constant too, every word p - 1
        mats.append(O.coset_lde_bitrev(t, lb, pow(7, hs[-1] // h, P)))
    zs = [(word(), word()), (word(), int(rng.integers(1, P - 1, dtype=np.uint64)))]
    alpha, beta = (word(), word()), (word(), word())
    dev = [product.to_device(m) for m in mats]
    ev = product.deep_evals(gpu_ctx, dev, lb, zs)
    assert np.array_equal(ev, O.deep_evals(mats, lb, zs))
    q = product.to_host(product.deep_quotient(gpu_ctx, dev, lb, alignment, zs, ev, alpha, beta))
    assert np.array_equal(q, O.deep_quotient(mats, lb, alignment, zs, ev, alpha, beta))


# about 700 leaves and as many compressions per level and proof: 16, 4 and 1
# lanes per compression; a warp, four lanes and a thread per leaf
@pytest.mark.parametrize("n", [2, 5, 40, 320])
def test_batches_of_every_size_match_single(product, gpu_ctx, n):
    k, t = O.cubic_trace(9, 12, 5)
    pcs = product.PcsParams(2, 1, 1, 3, 1, 100, 2)
    out = product.prove_multi(gpu_ctx, pcs, [product.AirWitness(product.AIR_CUBIC, t, k)])
    shapes = [product.AirShape(O.AIR_CUBIC, t.shape[0], t.shape[1], k)]
    f, c, d = out.proof.fields, out.proof.commitments, out.digest
    late_row, late_sibling = f.copy(), c.copy()
    late_row[-7] = (int(late_row[-7]) + 1) % P
    late_sibling[-1, 0] = (int(late_sibling[-1, 0]) + 1) % P
    variants = [(f, c, d), (late_row, c, d), (f, late_sibling, d), (f, c, d)]
    single = [product.verify_multi(gpu_ctx, pcs, shapes, *v).verdict for v in variants]
    assert single[0] == 0 and single[1] != 0 and single[2] != 0
    which = [0] * n
    which[0], which[n // 2], which[n - 1] = 1, 3, 2
    got, _ = product.verify_batch(gpu_ctx, [(pcs, shapes, *variants[w]) for w in which])
    assert got == [single[w] for w in which]
