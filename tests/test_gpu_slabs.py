"""A proof from a host trace, uploaded in column slabs that grow with the
height's rule (csrc/prover.cuh commit_main_pipelined), equals the proof from
the same trace on the device."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_h", [13, 14])
@pytest.mark.parametrize("width", [256, 700])
def test_host_trace_equals_device_trace(product, gpu_ctx, log_h, width):
    k, t = O.cubic_trace(log_h, width, log_h + width)
    pcs = product.PcsParams(1, 1, 0, 4, 0, 10, 0)
    host = product.prove_multi(gpu_ctx, pcs, [product.AirWitness(product.AIR_CUBIC, t, k)])
    dev = product.prove_multi(gpu_ctx, pcs, [product.AirWitness(product.AIR_CUBIC, product.to_device(t), k)])
    assert np.array_equal(host.digest, dev.digest)
    assert np.array_equal(host.proof.fields, dev.proof.fields)
    assert np.array_equal(host.proof.commitments, dev.proof.commitments)
