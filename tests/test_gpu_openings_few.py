"""Openings of few rows and digests (csrc/prover.cuh, gather_to_host): one and
two segments are copied, three and more gathered; rows that need padding, no
digest at all (every leaf opened), against the oracle's hints."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_h,widths,idx", [(0, [5], [0]), (0, [3, 8], [0]), (1, [20], [1]), (1, [20], [0, 1]),
                                              (2, [8], [2]), (2, [1, 9], [3]), (2, [7], [0, 2]), (3, [11], [5]),
                                              (3, [4, 4, 9], [0, 7]), (3, [6], list(range(8)))])
@pytest.mark.parametrize("alignment", [1, 8])
def test_few_segments(product, gpu_ctx, log_h, widths, idx, alignment):
    rng = np.random.default_rng(log_h + sum(widths))
    mats = [rng.integers(0, O.P, size=(1 << log_h, w), dtype=np.uint64) for w in widths]
    got = product.LmcsTree(gpu_ctx, [product.to_device(m) for m in mats], alignment).prove_batch(idx)
    want = O.OracleTree(O.default_p2(), mats, alignment).prove_batch(idx)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].reshape(-1), want[1].reshape(-1))
