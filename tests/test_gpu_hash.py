"""Trees of the sizes where the hash kernels change (16, 4 and 1 lanes per
state, csrc/merkle.cuh; the tensor-core permutation, csrc/p2tc.cuh), bit for
bit against the CPU oracle: block and round edges of the launches, rows that
end inside a chunk, several matrices and classes, extreme words and a
non-default permutation table."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P


def words(rng, h, w, kind):
    if kind == "top":  # every word at the top of the field
        return np.full((h, w), P - 1, dtype=np.uint64)
    m = rng.integers(0, P, size=(h, w), dtype=np.uint64)
    if kind == "edges":  # words around 2^32 multiples, where carries and borrows happen
        e = np.array([0, 1, 0xFFFFFFFF, 0x100000000, P - 1, P - 2, P - 0xFFFFFFFF, 1 << 63], dtype=np.uint64)
        m = e[rng.integers(0, len(e), size=(h, w))]
    return m


CASES = [
    ([(1 << 11, 9)], 8, "edges"),                        # the last class and level of 16 lanes per state
    ([(1 << 12, 17)], 8, "edges"),                       # four lanes per leaf
    ([(1 << 9, 4), (1 << 12, 8), (1 << 13, 13), (1 << 13, 1)], 8, "random"),  # carried states, two matrices
    ([(1 << 13, 3)], 1, "top"),
    ([(1 << 14, 12)], 8, "edges"),                       # the last class of four lanes per leaf
    ([(1 << 15, 1)], 1, "random"),                       # two groups per SM, one short chunk
    ([(1 << 15, 8)], 8, "top"),
    ([(1 << 15, 9)], 8, "edges"),                        # a chunk and one word
    ([(1 << 16, 25)], 8, "random"),                      # compression levels on the same path
    ([(1 << 12, 5), (1 << 15, 16), (1 << 15, 3)], 8, "edges"),  # carried states, two matrices in a class
    ([(1 << 14, 7), (1 << 16, 2)], 1, "random"),
    ([(1 << 18, 4)], 1, "edges"),                        # several rounds per CTA
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_large_trees_match_oracle(product, gpu_ctx, case):
    shapes, alignment, kind = CASES[case]
    rng = np.random.default_rng(500 + case)
    mats = [words(rng, h, w, kind) for h, w in shapes]
    ot = O.OracleTree(O.default_p2(), mats, alignment)
    gt = product.LmcsTree(gpu_ctx, [product.to_device(m) for m in mats], alignment)
    assert np.array_equal(gt.root(), ot.root())
    for l in (0, 1, 2):
        assert np.array_equal(gt.layer(l), ot.layer(l))


@pytest.mark.parametrize("diag", ["random", "small", "top"])
def test_large_tree_with_another_table_matches_oracle(product, diag):
    """The byte tables are built from the context's constants."""
    rng = np.random.default_rng(7)
    d = {"random": rng.integers(1, P, size=12, dtype=np.uint64), "small": np.arange(1, 13, dtype=np.uint64),
         "top": np.full(12, P - 1, dtype=np.uint64) - np.arange(12, dtype=np.uint64)}[diag]
    table = product.poseidon2_params_from_seed(99, d)
    m = words(rng, 1 << 15, 11, "edges")
    ctx = product.Context(0, table)
    try:
        gt = product.LmcsTree(ctx, [product.to_device(m)], 8)
        ot = O.OracleTree(O.p2_from_array(table), [m], 8)
        assert np.array_equal(gt.root(), ot.root())
        assert np.array_equal(gt.layer(0), ot.layer(0))
        del gt
    finally:
        ctx.close()


def test_openings_across_gather_chunks(product, gpu_ctx):
    """prove_batch gathers at most 2^24 words at a time: 2^14 rows of 1025
    words, padded to 1032, cross that line inside the row list."""
    rng = np.random.default_rng(3)
    m = rng.integers(0, P, size=(1 << 14, 1025), dtype=np.uint64)
    gt = product.LmcsTree(gpu_ctx, [product.to_device(m)], 8)
    fields, commits = gt.prove_batch(range(1 << 14))
    want = np.zeros((1 << 14, 1032), dtype=np.uint64)
    want[:, :1025] = m
    assert np.array_equal(fields.reshape(1 << 14, 1032), want)
    assert commits.shape[0] == 0
