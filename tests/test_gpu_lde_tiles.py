"""Coset LDE launches whose blocks take several column tiles (csrc/context.cuh,
tile_step): more than 148 x 2048 x 8 rows times tiles, so that a block reuses
its twiddle table and exchange buffer; every tile size as the top range and as
a pass, with a last turn that only some blocks take. Bit for bit against the
CPU oracle."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P


# split (low range first), width: 1200 tiles on 1184 blocks per group, 88 on 74, 50 on 37; a forward
# pass has half or a quarter as many blocks per group
@pytest.mark.parametrize("split,w,lb", [([5, 6], 9597, 1), ([6, 5], 9597, 1), ([7, 8], 701, 1), ([8, 7], 697, 1),
                                        ([9, 7], 395, 1), ([6, 10], 393, 1), ([10, 6], 400, 2), ([7, 9], 393, 1),
                                        ([5, 5, 5], 697, 1)])
def test_blocks_of_several_tiles(product, split, w, lb):
    L = sum(split)
    rng = np.random.default_rng(w + split[0])
    t = rng.integers(0, P, size=(1 << L, w), dtype=np.uint64)
    shift = int(rng.integers(1, P, dtype=np.uint64))
    ctx = product.Context(0)
    try:
        ctx.set_lde_split(L, split)
        got = product.to_host(product.coset_lde(ctx, product.to_device(t), lb, shift))
    finally:
        ctx.close()
    assert np.array_equal(got, O.coset_lde_bitrev(t, lb, shift))
