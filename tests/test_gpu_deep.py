"""DEEP evaluations over many matrices (csrc/prover.cuh, deep_evals): the
matrices are taken 24 to a launch (csrc/deep.cuh, MAX_DOTS), so the counts here
lie on both sides of one, two and the entry point's limit of 64."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu
P = O.P


@pytest.mark.parametrize("n", [23, 24, 25, 48, 49, 64])
def test_deep_evals_of_many_matrices(product, gpu_ctx, n):
    rng = np.random.default_rng(n)
    lb = 1
    log_h = np.sort(rng.integers(1, 8, size=n))
    log_h[-1] = 8
    widths = rng.choice([1, 3, 8, 17, 32, 33, 70], size=n)
    mats = [rng.integers(0, P, size=(1 << int(h), int(w)), dtype=np.uint64) for h, w in zip(log_h, widths)]
    zs = [tuple(int(x) for x in rng.integers(1, P, size=2, dtype=np.uint64)) for _ in range(2)]
    ev = product.deep_evals(gpu_ctx, [product.to_device(m) for m in mats], lb, zs)
    assert np.array_equal(ev, O.deep_evals(mats, lb, zs))


def test_deep_evals_of_many_heights(product):
    """26 heights: more folded weight vectors than one launch takes. A
    matrix's evaluations depend on it and on the tallest height only."""
    import torch
    gen = torch.Generator(device="cuda:0").manual_seed(3)
    word = lambda h: torch.randint(0, (1 << 63) - 1, (h, 1), generator=gen, device="cuda:0", dtype=torch.int64)
    mats = [word(1 << k) for k in range(26)]
    zs = [(5, 7), (11, 13)]
    ctx = product.Context(0)
    try:
        ev = product.deep_evals(ctx, mats, 0, zs)
        for k in (0, 1, 12, 23, 24):
            assert np.array_equal(ev[[k, 25]], product.deep_evals(ctx, [mats[k], mats[25]], 0, zs))
    finally:
        ctx.close()


def test_deep_evals_limit(product, gpu_ctx):
    m = product.to_device(np.ones((4, 1), dtype=np.uint64))
    with pytest.raises(product.P3gError):
        product.deep_evals(gpu_ctx, [m] * 65, 1, [(5, 7), (11, 13)])
