"""The proof-of-work search (csrc/fri.cuh) finds the least witness, also where
it lies turns of the grid away and where later candidates are given up midway;
against the CPU oracle's search."""
import ctypes as C

import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 8, 15, 17])
@pytest.mark.parametrize("n_pending", [0, 5, 7])
def test_least_witness(product, gpu_ctx, bits, n_pending):
    rng = np.random.default_rng(bits * 8 + n_pending)
    pp, lib = O.default_p2(), product.lib()
    for _ in range(4):
        ch = O.Challenger()
        O.lib().or_ch_init(C.byref(ch), C.byref(pp))
        for v in rng.integers(0, O.P, size=8 + n_pending, dtype=np.uint64):
            O.lib().or_ch_observe(C.byref(ch), int(v))
        state, pending = np.array(ch.state, dtype=np.uint64), np.array(ch.inp, dtype=np.uint64)
        assert ch.n_in == n_pending
        got = C.c_uint64()
        assert lib.p3g_grind(gpu_ctx.handle, O.ptr(state), O.ptr(pending), n_pending, bits, C.byref(got)) == 0
        assert got.value == O.lib().or_ch_grind(C.byref(ch), bits)
