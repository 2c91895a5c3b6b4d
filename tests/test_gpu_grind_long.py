"""Proof-of-work searches on both sides of the line where the grid widens
(csrc/fri.cuh, grind_grid): the least witness, against a search through the
permutation of plain batches of states."""
import ctypes as C

import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [21, 22])
def test_least_witness_of_a_long_search(product, gpu_ctx, bits):
    import torch
    rng = np.random.default_rng(bits)
    n = 1 << 20
    for _ in range(2):
        state = rng.integers(0, O.P, size=12, dtype=np.uint64)
        pending = rng.integers(0, O.P, size=3, dtype=np.uint64)
        got = C.c_uint64()
        assert product.lib().p3g_grind(gpu_ctx.handle, O.ptr(state), O.ptr(pending), 3, bits, C.byref(got)) == 0
        absorbed = state.copy()
        absorbed[:3] = pending
        first = None
        for base in range(0, got.value + 1, n):
            s = torch.from_numpy(absorbed.view(np.int64)).to("cuda:0").repeat(n, 1)
            s[:, 3] = torch.arange(base, base + n, device="cuda:0")
            product.poseidon2_permute_batch(gpu_ctx, s)
            hit = torch.nonzero((s[:, 7] & ((1 << bits) - 1)) == 0)
            if len(hit):
                first = base + int(hit[0, 0])
                break
        assert first == got.value
