"""Coset LDE kernels by bit range (csrc/lde.cuh): every tile size in each of
its roles (inverse pass, fused top range, forward pass), ranges below the
tile kernels', ragged and narrow widths, extreme words; bit for bit against
the CPU oracle."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P

CASES = [  # split (low range first), width, log_blowup
    ([5], 9, 1), ([6], 8, 2), ([7], 17, 1), ([8], 5, 3), ([9], 12, 1), ([10], 8, 1),  # fused range alone
    ([5, 5], 9, 2), ([5, 6], 8, 1), ([6, 5], 11, 3), ([7, 6], 8, 1), ([6, 7], 23, 1), ([8, 7], 9, 2),
    ([7, 8], 8, 1), ([9, 8], 10, 1), ([8, 9], 7, 1), ([10, 6], 8, 1), ([6, 10], 8, 2),
    ([5, 5, 5], 9, 1), ([6, 4, 5], 8, 1), ([4, 5], 8, 1), ([5, 4], 9, 1),             # generic kernels between
    ([7, 5], 3, 1), ([5, 6], 2, 2), ([8, 5], 4, 1),                                    # narrow tiles
    ([6, 6], 700, 1),                                                                  # several tiles per block
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("kind", ["random", "edges"])
def test_coset_lde_of_every_split(product, case, kind):
    split, w, lb = CASES[case]
    L = sum(split)
    rng = np.random.default_rng(case)
    t = rng.integers(0, P, size=(1 << L, w), dtype=np.uint64)
    if kind == "edges":
        e = np.array([0, 1, P - 1, P - 2, 0xFFFFFFFF, 0x100000000, 0xFFFF, P - 0xFFFF0000, 1 << 63, 0xFFFFFFFF00000000],
                     dtype=np.uint64)
        t = e[rng.integers(0, len(e), size=(1 << L, w))]
    shift = int(rng.integers(1, P, dtype=np.uint64))
    ctx = product.Context(0)
    try:
        ctx.set_lde_split(L, split)
        got = product.to_host(product.coset_lde(ctx, product.to_device(t), lb, shift))
    finally:
        ctx.close()
    assert np.array_equal(got, O.coset_lde_bitrev(t, lb, shift))
